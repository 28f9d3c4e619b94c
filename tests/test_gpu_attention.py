"""Decode attention on the tensor cores at the edges of its tiles, and prompt chunks against the same attention taken row by
row.  Oracle and tolerances are those of the other attention tests (crates/ksearch_kernels/src/lib.rs:1117-1237): q and p enter
as two f16 terms and K, V as exact integers with f32 scales, so the bound is that of f32 sums in another order."""
import numpy as np
import pytest

from ksearch_b200 import F16, F32, Eng, KsError, Q40, _lib, synth
from ksearch_b200 import model as ksm
from tests.test_gpu_ops import _attn_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act", [F32, F16])
@pytest.mark.parametrize("n_q,n_kv,hd", [(8, 1, 256), (8, 2, 256), (8, 4, 256), (8, 8, 256), (4, 2, 128), (8, 1, 128)])
def test_decode_attention_tile_edges(ctx, oracle, act, n_q, n_kv, hd):
    """Context lengths around the 16-position tiles and the 128-position splits, windows that start off a tile."""
    tlens = [1, 15, 16, 17, 127, 128, 129, 300]
    starts = [0, 0, 3, 0, 1, 0, 17, 83]
    for ns in (1, 3):
        _attn_case(ctx, oracle, Eng(act), len(tlens), n_q, n_kv, hd, 512, tlens, starts, hd ** -0.5, ns, act=act)


@pytest.mark.parametrize("act", [F32, F16])
@pytest.mark.parametrize("n_q,n_kv,hd", [(8, 2, 256), (4, 4, 128)])
def test_splits_dealt_by_length(ctx, oracle, act, n_q, n_kv, hd):
    """Slots of unequal contexts take splits by their lengths: sizes that fill the launch at once and sizes that need a spare chunk per
    slot, contexts of one position, the most slots, launches on either side of the two lines to the plain layout (contexts that average
    four fifths of the longest: 2000 and 1200, 1000 and 2200 over three; 128 positions a split: 512 in four), windows."""
    for tlens, ns in (([3000, 5], 2), ([1, 700, 129, 2048], 4), ([5, 6, 7, 1500, 9, 10, 11, 12], 3), ([1100] + [1 + 7 * i for i in range(31)], 4),
                      ([2000, 1600], 2), ([2000, 1599], 2), ([2000, 1200], 2), ([2000, 1199], 2), ([1000, 733, 733, 734], 4), ([1000, 733, 733, 733], 4), ([513, 1], 4), ([512, 1], 4), ([900, 16, 900, 100, 33], 5)):
        starts = [(11 * i) % 40 for i in range(len(tlens))]
        _attn_case(ctx, oracle, Eng(act), len(tlens), n_q, n_kv, hd, max(tlens) + 40, tlens, starts, hd ** -0.5, ns, act=act)


@pytest.mark.parametrize("hd,n_kv,window", [(256, 1, 0), (256, 2, 40), (128, 2, 0)])
def test_prompt_chunks_at_odd_sizes(ctx, oracle, hd, n_kv, window):
    """Chunks whose rows and positions end inside a tile, whole context and window: logits after the prompt match the CPU
    decoder's (the model's bound: 1e-3 of the logit scale)."""
    cfg = ksm.tiny_config(max_seq=320, n_kv=n_kv)
    cfg.hd = hd
    if window:
        cfg.sliding_window, cfg.swa_layers = window, 1
    model, T = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=31, keep=True)
    model.slot_alloc()
    toks = [int(t) for t in synth.token_ids(31, "p", 212, cfg.vocab)]
    cpu = oracle.CpuDecoder(oracle.decoder_cfg(cfg), T)
    at = 0
    for n in (3, 17, 65, 126):
        model.prefill(0, toks[at:at + n])
        for t in toks[at:at + n]:
            cpu.forward_token(t, False)
        at += n
    model.forward(0, 1, [toks[at]], True)
    ctx.synchronize()
    cpu.forward_token(toks[at], True)
    want, got = cpu.logits().astype(np.float64), model.read_debug(1, 0).astype(np.float64)
    assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
    cpu.close()
    model.close()


@pytest.mark.parametrize("n_q,n_kv", [(3, 1), (6, 1), (32, 1), (24, 2)])
@pytest.mark.parametrize("byte_off", [0, 2])
def test_head_groups_outside_the_set_are_refused(ctx, n_q, n_kv, byte_off):
    """1, 2, 4, 8 or 16 query heads per KV head, wherever the cache starts."""
    hd, max_t = 256, 64
    row = n_kv * hd // 32 * 18
    q, out, tmp = (ctx.buffer_empty_f32(n) for n in (n_q * hd, n_q * hd, 4))
    K, V, meta = ctx.buffer_empty_f32(max_t * row // 4 + 4), ctx.buffer_empty_f32(max_t * row // 4 + 4), ctx.buffer_bytes(np.array([9, 0, 0, 0], np.float32))
    before = ctx.launch_count()
    with pytest.raises(KsError) as ei:
        ctx.check(ctx.lib.ks_sdpa_decode(ctx.h, 1, n_q, n_kv, hd, max_t, Q40, 1.0, F32, q.h, K.h, V.h, byte_off, max_t * row, meta.h, tmp.h, out.h, 1))
    assert ei.value.code == _lib.ERR_UNSUPPORTED and ctx.launch_count() == before


@pytest.mark.parametrize("act", [F32, F16])
@pytest.mark.parametrize("hd,byte_off,pad", [(256, 4, 0), (256, 8, 0), (256, 0, 4), (128, 4, 0), (128, 0, 12), (256, 2, 0), (128, 0, 6)])
def test_caches_off_16_bytes(ctx, oracle, act, hd, byte_off, pad):
    """Caches that start, or follow one another, on 2, 4 or 8 bytes: the same answers as at 16, bit for bit on multiples of 4,
    where the same kernel takes them."""
    n_q, n_kv, max_t, scale, tlens, starts = 8, 2, 320, hd ** -0.5, [5, 280, 129], [2, 0, 40]
    npdt, n = np.float32 if act == F32 else np.float16, len(tlens)
    slot = max_t * n_kv * hd // 32 * 18
    K, V = (np.frombuffer(synth.q40_rows(53, k, n * max_t * n_kv * hd, sigma=0.05), np.uint8).reshape(n, slot) for k in "KV")
    q = synth.normals(53, "q", n * n_q * hd).astype(npdt)
    bq, meta = ctx.buffer_bytes(q), ctx.buffer_bytes(np.array([[t, s, 0, 0] for t, s in zip(tlens, starts)], np.float32))
    e = Eng(act)

    def run(off, gap, ns):
        def place(x):
            out = np.zeros(off + n * (slot + gap), np.uint8)
            out[off:].reshape(n, slot + gap)[:, :slot] = x
            return ctx.buffer_bytes(out)
        bK, bV, out = place(K), place(V), ctx.buffer_empty_bytes(q.nbytes)
        tmp = ctx.buffer_empty_f32(max(1, e.sdpa_tmp_floats(n_q, hd, ns, n)))
        ctx.check(ctx.lib.ks_sdpa_decode(ctx.h, n, n_q, n_kv, hd, max_t, Q40, scale, act, bq.h, bK.h, bV.h, off, slot + gap, meta.h, tmp.h, out.h, ns))
        return ctx.read_act(out, q.size, act).reshape(n, -1).astype(np.float64)

    for ns in (1, 3):
        got, plain = run(byte_off, pad, ns), run(0, 0, ns)
        if (byte_off | pad) % 4 == 0:
            assert np.array_equal(got, plain)
        for s in range(n):
            want = oracle.sdpa_decode(n_q, n_kv, hd, q.astype(np.float32).reshape(n, -1)[s], K[s], V[s], tlens[s], starts[s], scale, 0)
            rtol, atol = (1e-3, 1e-4) if act == F32 else (3e-3, 1e-3)
            assert (np.abs(got[s] - want) <= atol + rtol * np.abs(want)).all()


@pytest.mark.parametrize("act", [F32, F16])
@pytest.mark.parametrize("shape", ["tiny", "e2b_rows"])
@pytest.mark.parametrize("n", [65, 96, 97, 131, 145, 193, 256])
def test_prompt_chunks_in_blocks_of_either_size(ctx, oracle, act, shape, n):
    """65..256 prompt rows: every matrix of a layer reads its token rows in blocks of its own choice (wide ones, or several of up
    to 64), and the epilogues write the next matrix's.  The slot that took the rows in one chunk and one that took them 60 at a
    time leave the same next logits."""
    H, F, hd = (512, 1024, 128) if shape == "tiny" else (1536, 6144, 256)
    cfg = ksm.ModelConfig(2, H, F, 8, 1, hd, 2048, 320, 2, sigma_w=0.01 if act == F32 else 2e-5, sigma_embd=5e-5, act=act)
    model = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=33)
    toks = [int(t) for t in synth.token_ids(33, "p", n + 1, cfg.vocab)]
    got = []
    for slot, step in ((model.slot_alloc(), n), (model.slot_alloc(), 60)):
        for at in range(0, n, step):
            model.prefill(slot, toks[at:min(at + step, n)])
        model.forward(slot, 1, toks[n:], True)
        ctx.synchronize()
        got.append(model.read_debug(1, slot).astype(np.float64))
    # f32 sums in another order through two layers and 4-bit caches (the model's own bound); an f16 head rounds to 2^-11
    assert np.abs(got[0] - got[1]).max() <= (1e-3 if act == F32 else 2e-3) * np.abs(got[1]).max()
    model.close()


@pytest.mark.parametrize("n_q,n_kv,hd,window", [(4, 1, 128, 0), (8, 8, 128, 0), (8, 2, 256, 700)])
def test_prompt_rows_on_both_sides_of_the_sharing_rule(ctx, oracle, n_q, n_kv, hd, window):
    """Chunks whose rows take their context one by one, chunks that share it, and both again at other positions (the graph of a
    row count serves one form only): logits as the CPU decoder's after every chunk (the model's bound)."""
    cfg = ksm.tiny_config(max_seq=1600, n_kv=n_kv)
    cfg.n_q, cfg.hd, cfg.n_layers = n_q, hd, 2
    if window:
        cfg.sliding_window, cfg.swa_layers = window, 1
    model, T = ksm.GemmaCudaModel.synthetic(ctx, cfg, seed=34, keep=True)
    model.slot_alloc()
    toks = [int(t) for t in synth.token_ids(34, "p", 1500, cfg.vocab)]
    cpu = oracle.CpuDecoder(oracle.decoder_cfg(cfg), T)
    at = 0
    for n in (64, 20, 128, 200, 256, 256, 128, 20, 64, 200):
        model.prefill(0, toks[at:at + n])
        for t in toks[at:at + n]:
            cpu.forward_token(t, False)
        at += n
        model.forward(0, 1, [toks[at]], True)
        ctx.synchronize()
        cpu.forward_token(toks[at], True)
        at += 1
        want, got = cpu.logits().astype(np.float64), model.read_debug(1, 0).astype(np.float64)
        assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max(), (n, at)
    cpu.close()
    model.close()
