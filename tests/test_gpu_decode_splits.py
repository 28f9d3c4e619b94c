"""The persistent decode kernel where its attention changes form (one block per head, a few records merged by every block, many
by the head's last block) and at the widths its staging holds, against one launch per op on the same weights."""
import numpy as np
import pytest

from ksearch_b200 import CudaContext, synth
from ksearch_b200 import model as ksm

pytestmark = pytest.mark.gpu


def _logits(cfg, kernel, monkeypatch, toks, starts):
    monkeypatch.setenv("KSEARCH_DECODE_KERNEL", kernel)
    c = CudaContext(0, flags=1)
    m, _ = ksm.GemmaCudaModel.synthetic(c, cfg, seed=43, keep=True)
    m.slot_alloc()
    out = []
    for n in starts:
        m.slot_reset(0)
        if n:
            m.prefill(0, toks[:n])
        for t in toks[n:n + 4]:
            m.forward(0, 1, [t], True)
            c.synchronize()
            out.append(m.read_debug(1, 0).astype(np.float64))
    persistent = m.lib.ks_model_debug_ptr(m.h, 2, 0) is not None
    m.close()
    c.close()
    return out, persistent


@pytest.mark.parametrize("hidden,n_q,n_kv,hd,window", [
    (512, 4, 1, 128, 0), (512, 8, 8, 128, 0), (512, 8, 2, 256, 0), (512, 4, 2, 256, 90),
    (2048, 4, 1, 256, 0), (3584, 2, 1, 256, 0), (4096, 2, 2, 256, 0)])
def test_attention_forms_and_widths(monkeypatch, hidden, n_q, n_kv, hd, window):
    cfg = ksm.tiny_config(max_seq=1280, n_kv=n_kv)
    cfg.hidden, cfg.n_q, cfg.hd, cfg.n_layers = hidden, n_q, hd, 2
    if window:
        cfg.sliding_window, cfg.swa_layers = window, 0b01
    toks = [int(t) for t in synth.token_ids(43, "p", 1210, cfg.vocab)]
    starts = (0, 13, 57, 70, 86, 119, 240, 317, 1021, 1200)  # 60 | 61 positions and 320 | 321, and the window's edge
    got, persistent = _logits(cfg, "1", monkeypatch, toks, starts)
    assert persistent or window
    want, _ = _logits(cfg, "0", monkeypatch, toks, starts)
    for g, w in zip(got, want):
        scale, err = np.abs(w).max(), np.abs(g - w)
        assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale   # the bound of tests/test_gpu_model.py


@pytest.mark.parametrize("hidden,ffn,n_q,n_kv,hd,layers", [(512, 1024, 4, 1, 128, 18), (1536, 6144, 8, 1, 256, 3), (2560, 10240, 8, 2, 256, 9)])
def test_jobs_that_end_where_the_ring_ends(monkeypatch, hidden, ffn, n_q, n_kv, hd, layers):
    """Depths at which a run of weight rows fills the ring to its last byte (tests/test_decode_ring.py holds the places)."""
    cfg = ksm.tiny_config(max_seq=64, n_kv=n_kv)
    cfg.hidden, cfg.ffn, cfg.n_q, cfg.hd, cfg.n_layers, cfg.sigma_w = hidden, ffn, n_q, hd, layers, 2e-4
    toks = [int(t) for t in synth.token_ids(44, "p", 20, cfg.vocab)]
    got, persistent = _logits(cfg, "1", monkeypatch, toks, (0, 9))
    assert persistent
    want, _ = _logits(cfg, "0", monkeypatch, toks, (0, 9))
    for g, w in zip(got, want):
        scale, err = np.abs(w).max(), np.abs(g - w)
        assert err.max() <= 1e-3 * scale and np.sqrt((err ** 2).mean()) <= 1e-4 * scale
