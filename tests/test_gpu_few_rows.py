"""Matrices over 2..8 token rows on the tensor cores (mma.sync; the reference's batch matvec, crates/ksearch_kernels/src/lib.rs:1414),
and the edges of the tcgen05 kernels' tiles above that.  Held to the CPU dequant + dot of the GEMM tests: both operands keep f32
accuracy (exact weights, token rows as two f16 terms), so the bound is that of f32 sums in another order."""
import numpy as np
import pytest

from ksearch_b200 import Q4K, Q6K, CudaContext, KsError, _lib, synth
from tests.test_gpu_gemm import _check
from tests.test_gpu_matvec import _gen

pytestmark = pytest.mark.gpu


def _run(ctx, oracle, dtype, rows, cols, batch, launches=None):
    W = _gen(dtype, 95, f"W{rows}x{cols}", rows, cols)
    x = synth.normals(95, f"x{batch}", batch * cols).reshape(batch, cols).astype(np.float32)
    x[batch // 2] *= 3.0e4                                  # past the f16 range: its row carries a factor of its own
    y = ctx.buffer_empty_f32(batch * rows + 16)
    before = ctx.launch_count()
    bw, bx = ctx.buffer_bytes(W), ctx.buffer_bytes(x)
    ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, dtype, bw.h, 0, 0, bx.h, 0, y.h, 8, batch))
    if launches:
        assert ctx.launch_count() - before in launches
    got = ctx.read_f32(y, batch * rows + 16)
    assert not got[:8].any() and not got[8 + batch * rows:].any()
    y32, y64 = oracle.matvec(dtype, W, rows, cols, x)
    got, y32, y64 = got[8:8 + batch * rows].reshape(batch, rows), np.atleast_2d(y32), np.atleast_2d(y64)
    for t in range(batch):                                  # row by row: each has its own magnitude
        s = float(np.abs(x[t]).max())
        _check(got[t] / s, y32[t] / s, y64[t] / s, f"{rows}x{cols} row {t} of {batch}")


@pytest.mark.parametrize("rows,cols,batch", [
    (30001, 256, 2),      # one super-block: two warps a block, a last tile of one row
    (1003, 2560, 3),      # 20 warps, last tile of 11 rows
    (200, 11776, 3),      # 92 half super-blocks: no share of 4..20 warps but 4
    (520, 10240, 8),      # several column shares, partials summed by a second kernel
    (1010, 1536, 5), (16400, 512, 7),
])
def test_few_rows_q4k(ctx, oracle, rows, cols, batch):
    _run(ctx, oracle, Q4K, rows, cols, batch, (2, 3))       # operand split, GEMM, sum of the column shares


@pytest.mark.parametrize("rows,cols,batch", [
    (8008, 256, 2),       # two warps a block, last tile of 8 rows
    (1000, 1536, 3),      # twelve warps, two blocks per SM
    (1288, 2560, 8),      # the widest: 20 warps, one block per SM
    (2008, 1280, 4),      # five blocks a row: neighbouring rows differ in alignment
    (2007, 1280, 4),      # tiles that do not end on a 16-byte boundary: the tcgen05 kernel or the matvec
    (7001, 3072, 3),      # wider than a block
])
def test_few_rows_q6k(ctx, oracle, rows, cols, batch):
    _run(ctx, oracle, Q6K, rows, cols, batch)


@pytest.mark.parametrize("dtype,rows,cols", [(Q4K, 1000, 1536), (Q6K, 520, 512)])
@pytest.mark.parametrize("batch", [9, 16, 17, 32, 48, 64, 65, 96, 128, 129, 160, 256])
def test_gemm_token_tiles(ctx, oracle, dtype, rows, cols, batch):
    """Every step of the token-row tiling (one tile of up to 64, pairs of row tiles beyond, two token blocks beyond 128), over
    an odd count of row tiles."""
    _run(ctx, oracle, dtype, rows - 128 * (rows == 1000), cols, batch)


def test_gemm_blocks_at_the_ends_of_their_fields(ctx, oracle):
    """Super-blocks with d = 0, with dmin far above d, with all scales and minima 63 and with none."""
    rows, cols, batch = 130, 512, 24
    W = np.frombuffer(_gen(Q4K, 96, "Wend", rows, cols), np.uint8).reshape(rows, cols // 256, 144).copy()
    W[0::5, :, 0:2] = 0                                                     # d = 0
    W[1::5, :, 0:4] = np.frombuffer(np.array([1e-4, 0.05], np.float16).tobytes(), np.uint8)   # dmin = 500 d
    W[2::5, :, 4:16] = 255                                                  # sc = m = 63
    W[3::5, :, 4:16] = 0
    raw = W.tobytes()
    for n in (5, batch):
        x = synth.normals(96, f"x{n}", n * cols).reshape(n, cols).astype(np.float32)
        y = ctx.buffer_empty_f32(n * rows)
        bw, bx = ctx.buffer_bytes(np.frombuffer(raw, np.uint8)), ctx.buffer_bytes(x)
        ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, Q4K, bw.h, 0, 0, bx.h, 0, y.h, 0, n))
        y32, y64 = oracle.matvec(Q4K, np.frombuffer(raw, np.uint8), rows, cols, x)
        _check(ctx.read_f32(y, n * rows).reshape(n, rows), y32, y64, f"field ends, {n} rows")


def test_few_rows_wait_gives_up_and_recovers(oracle, monkeypatch):
    """The Q6_K kernel's tile of weights withheld: the bounded wait runs out, the status word reports it, the next call is right."""
    c = CudaContext(0, flags=1)
    rows, cols, batch = 2048, 1536, 4
    W = _gen(Q6K, 97, "Wstall", rows, cols)
    x = synth.normals(97, "xstall", batch * cols).reshape(batch, cols)
    bw, bx, y = c.buffer_bytes(W), c.buffer_bytes(x), c.buffer_empty_f32(batch * rows)
    monkeypatch.setenv("KSEARCH_GEMM_TEST_STALL", "1")
    c.check(c.lib.ks_matvec(c.h, rows, cols, Q6K, bw.h, 0, 0, bx.h, 0, y.h, 0, batch))
    with pytest.raises(KsError) as ei:
        c.synchronize()
    assert ei.value.code == _lib.ERR_TIMEOUT
    c.synchronize()
    monkeypatch.delenv("KSEARCH_GEMM_TEST_STALL")
    c.check(c.lib.ks_matvec(c.h, rows, cols, Q6K, bw.h, 0, 0, bx.h, 0, y.h, 0, batch))
    y32, y64 = oracle.matvec(Q6K, W, rows, cols, x)
    _check(c.read_f32(y, batch * rows).reshape(batch, rows), np.atleast_2d(y32), np.atleast_2d(y64), "after the give-up")
    c.close()
