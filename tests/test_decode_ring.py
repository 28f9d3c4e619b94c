"""Where the persistent decode kernel keeps its weights in shared memory: every job inside the ring, none on bytes that an older
one still holds, for every block of many shapes.  The places depend on the shape and the block alone, so this needs no GPU."""
import ctypes as C

import numpy as np
import pytest

from ksearch_b200 import _lib

SMS, SMEM = 148, 232448          # a B200: SMs, bytes of shared memory a block may have
E2B, E4B, TINY = (1536, 6144, 8, 1, 256), (2560, 10240, 8, 2, 256), (512, 1024, 4, 1, 128)


def _walk(lib, shape, layers, block):
    ring = C.c_uint(0)
    n = lib.ks_debug_decode_ring(*shape, layers, SMS, SMEM, block, C.byref(ring), None, 0)
    out = np.zeros((n, 3), np.uint32)
    assert lib.ks_debug_decode_ring(*shape, layers, SMS, SMEM, block, C.byref(ring), out.ctypes.data, n) == n
    return ring.value, out.astype(np.int64)


def _check(ring, jobs):
    at, size, oldest = jobs.T
    j = np.arange(len(jobs))
    assert (at % 16 == 0).all() and (at + size <= ring).all()
    assert (np.diff(oldest) >= 0).all() and (oldest <= j).all() and (j - oldest < 64).all()
    for back in range(1, 64):
        a, b = slice(back, None), slice(None, -back)
        live = j[b] >= oldest[a]
        clear = (at[a] + size[a] <= at[b]) | (at[b] + size[b] <= at[a])
        assert (clear | ~live).all()


def _all_blocks(lib, shape, layers):
    """Blocks with the same number of jobs in a layer do the same; they come in a few runs."""
    seen = {}
    for block in range(SMS):
        n = lib.ks_debug_decode_ring(*shape, 1, SMS, SMEM, block, None, None, 0)
        if n == 0:
            return 0
        groups = tuple(-(-(t - block) // SMS) if t > block else 0 for t in _groups(shape))
        if groups not in seen:
            seen[groups] = block
            _check(*_walk(lib, shape, layers, block))
    return len(seen)


def _groups(shape):
    h, f, nq, nkv, hd = shape
    return (nq * hd + 2 * nkv * hd) // 4, h // 4, f // 4


@pytest.mark.parametrize("shape", [E2B, E4B, TINY], ids=["e2b", "e4b", "tiny"])
def test_every_depth_of_the_configurations(shape):
    lib = _lib.load()
    for layers in range(1, 65):
        assert _all_blocks(lib, shape, layers) > 0


@pytest.mark.parametrize("hidden", range(512, 4097, 512))
def test_other_widths(hidden):
    lib = _lib.load()
    taken = 0
    for ffn in (2 * hidden, 3 * hidden, 4 * hidden, 8192, 14336, 30208):
        for nq, nkv, hd in ((2, 1, 256), (4, 4, 128), (8, 1, 256), (8, 8, 128), (16, 2, 128), (32, 8, 128)):
            for layers in (1, 2, 9, 18, 27, 30, 36, 42, 64, 128):
                taken += _all_blocks(lib, (hidden, ffn, nq, nkv, hd), layers) > 0
    assert taken >= 200
