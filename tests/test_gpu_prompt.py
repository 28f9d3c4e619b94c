"""Prompt chunks of up to 2048 rows against the same prompt in short pieces."""
import numpy as np
import pytest

from ksearch_b200 import F16, F32, synth
from ksearch_b200 import model as ksm

pytestmark = pytest.mark.gpu


def _logits_after(model, ctx, pieces, last):
    model.slot_reset(0)
    for p in pieces:
        model.prefill(0, p)
    model.forward(0, 1, [int(last)], True)
    ctx.synchronize()
    return model.read_debug(1, 0).astype(np.float64)


@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("n_kv", [1, 2])
def test_long_chunks_equal_short_pieces(ctx, n_kv, window):
    """One call with the whole prompt (chunks of up to 2048 rows: many blocks of token rows a launch, the rest behind a full
    chunk) and calls of 200 rows, which tests/test_gpu_model.py holds to the CPU decoder, leave the same cache: the next
    token's logits agree to the bound of those tests."""
    cfg = ksm.tiny_config(max_seq=2432, n_kv=n_kv)
    if window:
        cfg.sliding_window, cfg.swa_layers = window, 0b101
    model, _ = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=41, keep=True)
    model.slot_alloc()
    for n in (257, 640, 1025, 2047, 2048, 2049, 2051, 2400):
        toks = [int(t) for t in synth.token_ids(41, f"p{n}", n + 1, cfg.vocab)]
        want = _logits_after(model, ctx, [toks[i:min(i + 200, n)] for i in range(0, n, 200)], toks[n])
        got = _logits_after(model, ctx, [toks[:n]], toks[n])
        assert model.seq_len(0) == n + 1
        scale, err = np.abs(want).max(), np.abs(got - want)
        assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale, n
    model.close()


@pytest.mark.parametrize("n_q,n_kv,hd", [(8, 1, 256), (8, 2, 256), (4, 4, 256), (16, 1, 128), (8, 4, 128)])
def test_chunk_attention_equals_row_attention(monkeypatch, n_q, n_kv, hd):
    """Prompt rows that share their context (tiles of 128 query rows x 64 positions) against a model whose prompts go row by row
    through the decode attention: one tile and less, its edges, several tiles behind a context, windowed layers.  A pass that mixes
    slots always shares, so the piece brings a few rows of a second slot along."""
    from ksearch_b200 import CudaContext
    out = []
    for no_gemm in (False, True):
        if no_gemm:
            monkeypatch.setenv("KSEARCH_NO_GEMM", "1")
        else:
            monkeypatch.delenv("KSEARCH_NO_GEMM", raising=False)
        cfg = ksm.tiny_config(max_seq=768, n_slots=2, n_kv=n_kv)
        cfg.n_q, cfg.hd, cfg.n_layers = n_q, hd, 2
        cfg.sliding_window, cfg.swa_layers = 70, 0b10
        c = CudaContext(0, flags=1)
        model, _ = ksm.GemmaCudaModel.synthetic(c, cfg, seed=47, keep=True)
        slots = [model.slot_alloc(), model.slot_alloc()]
        toks = [int(t) for t in synth.token_ids(47, "p", 700, cfg.vocab)]
        for first, n in ((0, 1), (0, 63), (0, 64), (0, 129), (0, 333), (65, 128), (300, 257), (600, 90)):
            for s in slots:
                model.slot_reset(s)
            if first:
                model.prefill(0, toks[:first])
            model.prefill_many([(0, toks[first:first + n]), (1, toks[:5])])
            model.forward(0, 2, [toks[first + n], toks[5]], True)
            c.synchronize()
            out.append(np.concatenate([model.read_debug(1, s).astype(np.float64) for s in slots]))
        model.close()
        c.close()
    half = len(out) // 2
    for got, want in zip(out[:half], out[half:]):
        scale, err = np.abs(want).max(), np.abs(got - want)
        assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale


@pytest.mark.parametrize("n_kv,window", [(1, 0), (2, 60)])
def test_prompts_of_several_slots_share_passes(ctx, n_kv, window):
    """prefill_many against one prefill call per slot: ragged pieces in any slot order, pieces behind a context, an empty one, more
    rows than a pass takes; what is refused leaves every slot where it was."""
    from ksearch_b200 import KsError
    cfg = ksm.tiny_config(max_seq=800, n_slots=4, n_kv=n_kv)
    cfg.sliding_window, cfg.swa_layers = window, 0b101 if window else 0
    model, _ = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=53, keep=True)
    slots = [model.slot_alloc() for _ in range(4)]
    toks = [[int(t) for t in synth.token_ids(53, f"s{s}", 801, cfg.vocab)] for s in slots]
    for rounds in ([(5, 130, 1, 300)], [(64, 17, 128, 3), (1, 1, 0, 1), (90, 0, 257, 40)], [(700, 690, 710, 705)]):
        logits = []
        for together in (True, False):
            at = [0] * 4
            for s in slots:
                model.slot_reset(s)
            for counts in rounds:
                parts = [(s, toks[s][at[s]:at[s] + counts[s]]) for s in (2, 0, 3, 1)]
                if together:
                    model.prefill_many(parts)
                else:
                    for s, p in parts:
                        model.prefill(s, p)
                at = [a + c for a, c in zip(at, counts)]
            assert [model.seq_len(s) for s in slots] == at
            model.forward(0, 4, [toks[s][at[s]] for s in slots], True)
            ctx.synchronize()
            logits.append([model.read_debug(1, s).astype(np.float64) for s in slots])
        for got, want in zip(*logits):
            scale, err = np.abs(want).max(), np.abs(got - want)
            assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale
    before = [model.seq_len(s) for s in slots]
    for bad in ([(0, [1]), (1, [cfg.vocab])], [(0, [1]), (0, [2])], [(0, [1]), (1, [1] * 800)]):
        with pytest.raises(KsError):
            model.prefill_many(bad)
        assert [model.seq_len(s) for s in slots] == before
    model.close()


def test_lengths_that_do_not_repeat_leave_no_graph(ctx):
    """A prompt length is launched the first time, captured the second and replayed from then on, always with the same result; lengths
    that come once leave nothing behind, and what repeated ones leave is bounded."""
    cfg = ksm.tiny_config(max_seq=1280)
    model, _ = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=59, keep=True)
    model.slot_alloc()
    toks = [int(t) for t in synth.token_ids(59, "p", 1280, cfg.vocab)]
    held = lambda: model.lib.ks_model_debug_graphs(model.h)
    first = {n: _logits_after(model, ctx, [toks[:n]], toks[n]) for n in (9, 130, 700, 1100)}   # (the decode step is a graph)
    before = held()
    for n in range(20, 220):
        model.slot_reset(0)
        model.prefill(0, toks[:n])
    assert held() == before
    for _ in range(3):
        for n, want in first.items():
            assert np.array_equal(_logits_after(model, ctx, [toks[:n]], toks[n]), want), n
    assert held() == before + len(first)
    for n in range(300, 400):
        for _ in range(2):
            model.slot_reset(0)
            model.prefill(0, toks[:n])
    assert held() == before + 64
    for n, want in first.items():
        assert np.array_equal(_logits_after(model, ctx, [toks[:n]], toks[n]), want), n
    assert held() <= before + 64
    model.close()


@pytest.mark.parametrize("window", [0, 100])
def test_equal_pieces_of_a_growing_prompt(ctx, window):
    """Pieces of one length behind each other, three prompts: their passes are launched, captured and replayed while the context grows
    past what the first of them saw.  The same logits every time, and those of shorter pieces to the bound above."""
    cfg = ksm.tiny_config(max_seq=5000, n_kv=2)
    if window:
        cfg.sliding_window, cfg.swa_layers = window, 0b101
    model, _ = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=71, keep=True)
    model.slot_alloc()
    toks = [int(t) for t in synth.token_ids(71, "p", 4097, cfg.vocab)]
    got = [_logits_after(model, ctx, [toks[i:i + 512] for i in range(0, 4096, 512)], toks[4096]) for _ in range(3)]
    want = _logits_after(model, ctx, [toks[i:min(i + 200, 4096)] for i in range(0, 4096, 200)], toks[4096])
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    scale, err = np.abs(want).max(), np.abs(got[0] - want)
    assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale
    model.close()


@pytest.mark.parametrize("n_slots,n_kv,hd,act,window", [(4, 2, 256, F32, 60), (4, 1, 256, F16, 0), (4, 2, 128, F16, 40), (12, 1, 128, F32, 50), (64, 1, 128, F32, 0)])
def test_mixed_passes_of_other_models(ctx, n_slots, n_kv, hd, act, window):
    """prefill_many against one prefill call per slot: head size 256, f16 activations, up to as many slots as a model has.  In f16 both
    sides run the prompt in f32; the step behind it rounds to f16 (2^-11 an op, ten ops a layer, three layers)."""
    cfg = ksm.tiny_config(max_seq=256, n_slots=n_slots, n_kv=n_kv, act=act)
    cfg.hd = hd
    if act == F16:
        cfg.sigma_w = 3e-5   # random weights of one sign: larger ones leave the f16 range in the FFN
    if window:
        cfg.sliding_window, cfg.swa_layers = window, 0b101
    model, _ = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=61, keep=True)
    slots = [model.slot_alloc() for _ in range(n_slots)]
    toks = [[int(t) for t in synth.token_ids(61, f"s{s}", 256, cfg.vocab)] for s in slots]
    rounds = [[(7 * s) % 61 + 1 for s in slots], [(11 * s) % 19 for s in slots]]
    sides = []
    for together in (True, False):
        at = [0] * n_slots
        for s in slots:
            model.slot_reset(s)
        for counts in rounds:
            parts = [(s, toks[s][at[s]:at[s] + counts[s]]) for s in reversed(slots)]
            if together:
                model.prefill_many(parts)
            else:
                for s, p in parts:
                    model.prefill(s, p)
            at = [a + c for a, c in zip(at, counts)]
        model.forward(0, n_slots, [toks[s][at[s]] for s in slots], True)
        ctx.synchronize()
        sides.append([model.read_debug(1, s).astype(np.float64) for s in slots])
    worst, mean = (1e-3, 1e-4) if act == F32 else (30 * 2.0 ** -11, 30 ** 0.5 * 2.0 ** -11)
    for got, want in zip(*sides):
        scale, err = np.abs(want).max(), np.abs(got - want)
        assert 0 < scale < np.inf
        assert err.max() <= worst * scale and np.sqrt((err ** 2).mean()) <= mean * scale
    model.close()


@pytest.mark.parametrize("ffn", [2304, 3328, 16384])
def test_gelu_of_four_rows_per_cluster(ctx, oracle, ffn):
    """From 128 rows and 2^18 values on four token rows share a cluster of blocks: row counts around a multiple of four, widths that
    leave warps of a block and blocks of the cluster without work, the widest rows.  Against pieces of 100 rows, which have a cluster per row,
    and against the CPU decoder: the model's bounds."""
    cfg = ksm.ModelConfig(2, 256, ffn, 2, 1, 128, 1024, 256, 1, sigma_w=0.01, sigma_embd=1e-4)
    model, T = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=43, keep=True)
    model.slot_alloc()
    toks = [int(t) for t in synth.token_ids(43, "p", 200, cfg.vocab)]
    for n in (128, 129, 130, 131, 191):
        want = _logits_after(model, ctx, [toks[i:min(i + 100, n)] for i in range(0, n, 100)], toks[n])
        got = _logits_after(model, ctx, [toks[:n]], toks[n])
        scale, err = np.abs(want).max(), np.abs(got - want)
        assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale, n
    cpu = oracle.CpuDecoder(oracle.decoder_cfg(cfg), T)
    for t in toks[:n + 1]:
        cpu.forward_token(t, True)
    want = cpu.logits().astype(np.float64)
    scale, err = np.abs(want).max(), np.abs(got - want)
    assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale
    cpu.close()
    model.close()


@pytest.mark.parametrize("window", [0, 100])
def test_prompts_of_a_model_without_decoded_tiles(ctx, monkeypatch, window):
    """A model that has no memory for decoded tiles takes prompts row by row and slots one by one: the same logits to the model's bound,
    behind one prompt, pieces of it and pieces of several slots."""
    cfg = ksm.tiny_config(max_seq=1280, n_slots=3, n_kv=2)
    if window:
        cfg.sliding_window, cfg.swa_layers = window, 0b101
    toks = [int(t) for t in synth.token_ids(73, "p", 1280, cfg.vocab)]
    out = []
    for image in ("1", "0"):
        monkeypatch.setenv("KSEARCH_KV_IMAGE", image)
        model, _ = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=73, keep=True)
        slots = [model.slot_alloc() for _ in range(3)]
        got = [_logits_after(model, ctx, p, toks[0]) for p in ([toks[:1200]], [toks[:1200]], [toks[:1200]], [toks[:700], toks[700:1200]])]
        for s in slots:
            model.slot_reset(s)
        for _ in range(2):
            model.prefill_many([(s, toks[100 * s:100 * s + 150 + 90 * s]) for s in slots])
        model.forward(0, 3, toks[:3], True)
        ctx.synchronize()
        out.append(got + [model.read_debug(1, s).astype(np.float64) for s in slots])
        assert [model.seq_len(s) for s in slots] == [2 * (150 + 90 * s) + 1 for s in slots]
        model.close()
    for want, got in zip(*out):
        scale, err = np.abs(want).max(), np.abs(got - want)
        assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale


def test_mixed_pass_with_more_context_than_its_decoded_tiles(ctx):
    """Eight slots of 15 tiles of 64 positions and 32 KV heads are more than the 63 tiles such a model keeps decoded (256 MB, 4 MB and a word per head each): their short
    pieces run in several passes.  Against the same pieces one by one, whose rows read the caches themselves: the model's bound."""
    cfg = ksm.ModelConfig(1, 256, 512, 32, 32, 256, 1024, 1024, 8, sigma_w=0.01, sigma_embd=1e-4)
    model, _ = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=53, keep=True)
    slots = [model.slot_alloc() for _ in range(8)]
    toks = [int(t) for t in synth.token_ids(53, "p", 1000, cfg.vocab)]
    out = []
    for together in (True, False):
        for s in slots:
            model.slot_reset(s)
            model.prefill(s, toks[s:s + 900])
        pieces = [(s, toks[s:s + 5 + s]) for s in slots]
        if together:
            model.prefill_many(pieces)
        else:
            for s, p in pieces:
                model.prefill(s, p)
        model.forward(0, 8, toks[:8], True)
        ctx.synchronize()
        out.append(np.concatenate([model.read_debug(1, s).astype(np.float64) for s in slots]))
    scale, err = np.abs(out[1]).max(), np.abs(out[0] - out[1])
    assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale
    model.close()
