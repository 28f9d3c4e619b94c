"""Attention of prompt rows that share their context (128 query rows x 64 positions a tile) alone, against 64 bits: rows and
positions that end inside a tile, windows shorter and longer than one, several parts in one launch, empty splits.

q and the probabilities are two f16 terms, K and V exact as two; what is left out of a product or rounded off is 2^-22 of it at
most, at random signs.  In a score that adds up to 2^-22 of the 2-norm of its products, which is what the probability is off by; the
values add 2^-22 twice.  So the bound on the result's 2-norm is 2^-22 (2 + the largest such norm), about 7e-7 where scores are of
about 1, with f32 sums and exponentials (2^-24 a step) inside that."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(blocks, hd):
    b = blocks.reshape(-1, hd // 32, 18)
    d = b[:, :, :2].copy().view(np.float16).astype(np.float64)
    n = b[:, :, 2:].astype(np.int64)
    return (np.concatenate([(n & 15) - 8, (n >> 4) - 8], 2) * d).reshape(-1, hd)


def _cache(rng, positions, n_kv, hd, scale):
    n = positions * n_kv * hd // 32
    b = np.empty((n, 18), np.uint8)
    b[:, 2:] = rng.integers(0, 256, (n, 16))
    b[:, :2] = scale(n).astype(np.float16).view(np.uint8).reshape(n, 2)
    return b


def _run(ctx, n_q, n_kv, hd, parts, window, n_splits, k_scale=None, q_sigma=1.0):
    """parts: (positions in front, rows) of each slot.  Per part: the result, what 64 bits give, the bound."""
    rng = np.random.default_rng(n_q * 1000 + n_kv * 100 + hd + window + n_splits)
    max_t = max(b + n for b, n in parts) + 3
    small = lambda n: np.abs(rng.standard_normal(n)) * 0.1
    K, V = (_cache(rng, max_t * len(parts), n_kv, hd, s) for s in (k_scale or small, small))
    rows = sum(n for _, n in parts)
    q = (rng.standard_normal((rows, n_q, hd)) * q_sigma).astype(np.float32)
    row0 = np.cumsum([0] + [n for _, n in parts])
    slots = list(range(len(parts)))[::-1]      # any order
    ends = np.concatenate([np.arange(b + 1, b + n + 1) for b, n in parts])
    first = np.maximum(ends - window, 0) if window else np.zeros_like(ends)
    meta = np.zeros((rows, 4), np.float32)
    meta[:, 0], meta[:, 1] = ends - first, first
    scale = hd ** -0.5
    tmp = ctx.buffer_bytes(np.full((rows, n_q, n_splits, hd + 2), np.nan, np.float32))
    keep = [ctx.buffer_bytes(a) for a in (q, K, V, meta)]
    stride = max_t * n_kv * hd // 32 * 18
    ctx.check(ctx.lib.ks_debug_sdpa_chunk(ctx.h, n_q, n_kv, hd, max_t, scale, len(parts), (C.c_int * len(row0))(*row0.tolist()), (C.c_int * len(slots))(*slots),
                                          stride, keep[0].h, keep[1].h, keep[2].h, keep[3].h, tmp.h, n_splits))
    rec = ctx.read_f32(tmp, rows * n_q * n_splits * (hd + 2)).reshape(rows, n_q, n_splits, hd + 2).astype(np.float64)
    m, l, o = rec[..., 0], rec[..., 1], rec[..., 2:]
    f = np.where(l != 0, np.exp(m - m.max(2, keepdims=True)), 0)     # an empty split may leave no values
    got = (np.where(l[..., None] != 0, o, 0) * f[..., None]).sum(2) / (np.where(l != 0, l, 0) * f).sum(2)[..., None]
    Kd, Vd = (_values(a, hd).reshape(len(parts), max_t, n_kv, hd) for a in (K, V))
    want, spread = np.empty_like(got), np.zeros(len(parts))
    for p, slot in enumerate(slots):
        r = slice(row0[p], row0[p + 1])
        seen = (np.arange(max_t) < ends[r, None]) & (np.arange(max_t) >= first[r, None])
        for h in range(n_q):
            s = np.where(seen, q[r, h].astype(np.float64) @ Kd[slot, :, h // (n_q // n_kv)].T * scale, -np.inf)
            products = (q[r, h].astype(np.float64) ** 2) @ (Kd[slot, :, h // (n_q // n_kv)] ** 2).T
            spread[p] = max(spread[p], np.sqrt(np.where(seen, products, 0).max()) * scale)
            e = np.exp(s - s.max(1, keepdims=True))
            want[r, h] = e @ Vd[slot, :, h // (n_q // n_kv)] / e.sum(1, keepdims=True)
    return [(got[row0[p]:row0[p + 1]], want[row0[p]:row0[p + 1]], 2.0 ** -22 * (2 + spread[p])) for p in range(len(parts))]


def _hold(pairs):
    for p, (got, want, bound) in enumerate(pairs):
        assert np.isfinite(got).all(), p
        assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want), p


@pytest.mark.parametrize("window", [0, 33, 64, 100])
@pytest.mark.parametrize("n_q,n_kv,hd", [(8, 1, 256), (8, 2, 256), (4, 4, 256), (16, 1, 256), (16, 1, 128), (8, 4, 128), (8, 8, 128)])
def test_parts_at_tile_edges(ctx, n_q, n_kv, hd, window):
    parts = [(0, 1), (0, 15), (40, 16), (3, 17), (64, 63), (200, 64), (129, 65), (0, 129), (511, 2), (63, 1)]
    for n_splits in (1, 3):
        _hold(_run(ctx, n_q, n_kv, hd, parts, window, n_splits))


@pytest.mark.parametrize("n_q,n_kv,hd", [(8, 1, 256), (8, 2, 256), (4, 1, 128)])
def test_error_does_not_grow_with_the_context(ctx, n_q, n_kv, hd):
    _hold(_run(ctx, n_q, n_kv, hd, [(3900, 70)], 0, 1))
    _hold(_run(ctx, n_q, n_kv, hd, [(0, 700)], 0, 5))


@pytest.mark.parametrize("n_q,n_kv,hd", [(8, 1, 256), (8, 4, 128)])
def test_keys_of_any_f16_scale(ctx, n_q, n_kv, hd):
    """Scales whose products leave f16 in some tiles and rows, ordinary ones beside them; the largest finite one."""
    rng = np.random.default_rng(5)

    def scale(n):
        big = np.repeat(rng.random(-(-n // 16)) < 0.1, 16)[:n] & (rng.random(n) < 0.5)
        return np.where(big, rng.choice([8189.0, 9000.0, 20000.0, 65504.0], n), np.abs(rng.standard_normal(n)) * 100)

    _hold(_run(ctx, n_q, n_kv, hd, [(0, 65), (300, 40), (64, 64)], 0, 2, scale, 1e-5))


def test_many_parts(ctx):
    """As many parts as a launch takes, one row each among longer ones."""
    _hold(_run(ctx, 8, 1, 256, [(i * 3 % 90, 1 + (i * 7) % 19) for i in range(64)], 0, 2))
