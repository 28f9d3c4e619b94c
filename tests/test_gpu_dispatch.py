"""Calls at the edges of the dispatch: what the fast kernels do not take has to reach the kernel that does, or be refused on
the host.  Oracle and bounds are those of the op's own tests."""
import ctypes as C

import numpy as np
import pytest

from ksearch_b200 import Q4K, Q6K, CudaContext, KsError, _lib, synth
from tests.test_gpu_gemm import _check
from tests.test_gpu_matvec import _gen

pytestmark = pytest.mark.gpu


def _view(ctx, buf, byte_off):
    """The library's handle of a caller's memory that starts byte_off bytes into buf."""
    return ctx.lib.ks_buf_wrap(ctx.h, buf.ptr + byte_off, buf.nbytes - byte_off)


@pytest.mark.parametrize("dtype,rows,cols,batch", [(Q4K, 4096, 1536, 3), (Q6K, 2048, 1536, 3), (Q4K, 4096, 512, 8)])
def test_few_rows_off_16_bytes(ctx, oracle, dtype, rows, cols, batch):
    """Shapes whose 2..8 token rows go through the GEMM when they start on 16 bytes.  Where they do not (a wrapped buffer, an
    odd element offset), the batch matvec takes the call in its one launch; a batch of more than 8 is refused."""
    W = _gen(dtype, 71, "W", rows, cols)
    x = synth.normals(71, "x", 9 * cols).reshape(9, cols).astype(np.float32)
    bw, y = ctx.buffer_bytes(W), ctx.buffer_empty_f32(9 * rows)
    bx = ctx.buffer_bytes(np.concatenate([np.zeros(4, np.float32), x.ravel(), np.zeros(4, np.float32)]))
    y32, y64 = oracle.matvec(dtype, W, rows, cols, x[:batch])
    for floats, x_off, launches in ((4, 0, (2, 3)), (3, 1, (2, 3)), (1, 3, (2, 3)), (0, 4, (2, 3))):   # all of them name x itself
        h = _view(ctx, bx, 4 * floats)
        before = ctx.launch_count()
        ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, dtype, bw.h, 0, 0, h, x_off, y.h, 0, batch))
        assert ctx.launch_count() - before in launches
        _check(ctx.read_f32(y, batch * rows).reshape(batch, rows), y32, y64, f"view at {floats} floats, offset {x_off}")
        ctx.lib.ks_buf_free(ctx.h, h)
    moved = ctx.buffer_bytes(np.concatenate([np.zeros(5, np.float32), x.ravel()]))                     # x at 20 bytes past a 256-byte boundary
    for floats, x_off in ((5, 0), (0, 5), (1, 4)):
        h = _view(ctx, moved, 4 * floats)
        before = ctx.launch_count()
        ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, dtype, bw.h, 0, 0, h, x_off, y.h, 0, batch))
        assert ctx.launch_count() - before == 1
        _check(ctx.read_f32(y, batch * rows).reshape(batch, rows), y32, y64, f"view at {floats} floats, offset {x_off}")
        with pytest.raises(KsError) as ei:
            ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, dtype, bw.h, 0, 0, h, x_off, y.h, 0, 9))
        assert ei.value.code == _lib.ERR_INVALID
        ctx.lib.ks_buf_free(ctx.h, h)


@pytest.mark.parametrize("dtype,byte_off", [(Q4K, 8), (Q6K, 1)])
@pytest.mark.parametrize("batch", [1, 3, 9])
def test_weights_off_their_alignment_are_refused(ctx, dtype, byte_off, batch):
    """Q4_K rows start on 16 bytes, Q6_K rows on 2: a wrapped buffer that starts elsewhere is refused before any launch."""
    rows, cols = 2048, 1536
    W = _gen(dtype, 72, "W", rows, cols)
    bw = ctx.buffer_bytes(np.concatenate([np.zeros(16, np.uint8), np.frombuffer(W, np.uint8)]))
    bx, y = ctx.buffer_empty_f32(batch * cols), ctx.buffer_empty_f32(batch * rows)
    h = _view(ctx, bw, byte_off)
    before = ctx.launch_count()
    with pytest.raises(KsError) as ei:
        ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, dtype, h, 0, 0, bx.h, 0, y.h, 0, batch))
    assert ei.value.code == _lib.ERR_INVALID and ctx.launch_count() == before
    ctx.lib.ks_buf_free(ctx.h, h)


@pytest.mark.parametrize("dtype,op", [(Q4K, "mv_q4k"), (Q6K, "mv_q6k")])
@pytest.mark.parametrize("batch", [3, 8])
def test_plans_speak_for_few_rows_too(oracle, dtype, op, batch):
    """A shape whose 3..8 token rows go through the GEMM by themselves: with an override, or a plan stored for that row count,
    the matvec kernel the plan names runs (one launch), whatever the other row counts do."""
    rows, cols = 4096, 1536
    c = CudaContext(0)
    W = _gen(dtype, 73, "W", rows, cols)
    x = synth.normals(73, "x", batch * cols).reshape(batch, cols).astype(np.float32)
    bw, bx, y = c.buffer_bytes(W), c.buffer_bytes(x), c.buffer_empty_f32(batch * rows)
    y32, y64 = oracle.matvec(dtype, W, rows, cols, x)

    def launches(n=batch):
        before = c.launch_count()
        c.check(c.lib.ks_matvec(c.h, rows, cols, dtype, bw.h, 0, 0, bx.h, 0, y.h, 0, n))
        _check(c.read_f32(y, n * rows).reshape(n, rows), y32[:n], y64[:n], f"{op} x {n}")
        return c.launch_count() - before

    assert launches() > 1
    for variant in (0, 1):
        plan = _lib.Plan(variant=variant, nr=1 if variant == 0 else 2, nwarps=4, ctas_per_sm=2, ms=0.0)
        c.check(c.lib.ks_plan_override(c.h, C.byref(plan)))
        assert launches() == 1
        c.check(c.lib.ks_plan_override(c.h, None))
        assert launches() > 1
        c.check(c.lib.ks_plan_set(c.h, op.encode(), rows, cols, batch, C.byref(plan)))
        assert launches() == 1 and (batch == 3 or launches(batch - 1) > 1)
        c.check(c.lib.ks_plan_set(c.h, op.encode(), rows, cols, batch, None))
    assert launches() > 1
    c.close()


def _blocks_of(c, call):
    """Blocks of the one launch that a call captures to on the context's stream."""
    from cuda.bindings import driver as cu
    stream = cu.CUstream(c.lib.ks_ctx_stream(c.h))
    (err,) = cu.cuStreamBeginCapture(stream, cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL)
    assert err == cu.CUresult.CUDA_SUCCESS
    try:
        call()
    finally:
        err, graph = cu.cuStreamEndCapture(stream)
    assert err == cu.CUresult.CUDA_SUCCESS
    err, _, n = cu.cuGraphGetNodes(graph)
    err, nodes, n = cu.cuGraphGetNodes(graph, n)
    assert err == cu.CUresult.CUDA_SUCCESS and n == 1
    err, at = cu.cuGraphKernelNodeGetParams(nodes[0])
    assert err == cu.CUresult.CUDA_SUCCESS
    blocks, threads = at.gridDimX, at.blockDimX
    cu.cuGraphDestroy(graph)
    return blocks, threads


def test_a_plan_without_warps_keeps_its_other_fields(oracle):
    """nwarps 0 in a plan is the kernel's default for that field and no more: its blocks per SM stand.  Without a plan the launch is
    the shape's own."""
    rows, cols = 20480, 1536
    c = CudaContext(0)
    sms = c.lib.ks_ctx_sm_count(c.h)
    W, x = _gen(Q4K, 78, "W", rows, cols), synth.normals(78, "x", cols).astype(np.float32)
    bw, bx, y = c.buffer_bytes(W), c.buffer_bytes(x), c.buffer_empty_f32(rows)
    y32, y64 = oracle.matvec(Q4K, W, rows, cols, x)

    def call():
        c.check(c.lib.ks_matvec(c.h, rows, cols, Q4K, bw.h, 0, 0, bx.h, 0, y.h, 0, 1))

    def launch(plan):
        for how in ("override", "set"):
            if how == "override":
                c.check(c.lib.ks_plan_override(c.h, C.byref(plan)))
            else:
                c.check(c.lib.ks_plan_set(c.h, b"mv_q4k", rows, cols, 1, C.byref(plan)))
            got = _blocks_of(c, call)
            call()
            _check(c.read_f32(y, rows), y32, y64, how)
            c.check(c.lib.ks_plan_override(c.h, None))
            c.check(c.lib.ks_plan_set(c.h, b"mv_q4k", rows, cols, 1, None))
            yield got

    own = _blocks_of(c, call)
    for per_sm in (1, 2, 3):
        for blocks, threads in launch(_lib.Plan(variant=0, nr=1, nwarps=0, ctas_per_sm=per_sm, ms=0.0)):
            assert blocks == min(sms * per_sm, -(-rows // 4 // (threads // 32)))
    for blocks, threads in launch(_lib.Plan(variant=0, nr=1, nwarps=6, ctas_per_sm=1, ms=0.0)):
        assert (blocks, threads) == (sms, 192)
    assert _blocks_of(c, call) == own
    c.close()


@pytest.mark.parametrize("gate_up,cols,per_sm,warps", [
    (0, 2560, 2.5, 4), (0, 3584, 1.5, 4), (0, 3584, 3, 8), (0, 2560, 7.9, 8), (1, 1536, 1.9, 4), (1, 1536, 7.9, 8),     # few groups of four rows
    (0, 2560, 8.1, 6), (0, 2560, 12, 6), (0, 2560, 12.1, 8), (0, 2560, 17, 8), (0, 3584, 17, 8), (0, 3584, 20, 8), (0, 2560, 20.1, 6), (0, 3584, 24, 6), (0, 2560, 28, 8), (0, 3584, 34, 8),
    (0, 1024, 10, 8), (0, 1024, 13, 8), (0, 1024, 22, 6), (0, 1024, 25, 8), (0, 2048, 13, 8),
    (1, 3584, 9, 6), (1, 3584, 15, 8), (1, 3584, 19, 8), (1, 3584, 22, 6), (1, 3584, 32, 8), (1, 1024, 10, 8), (1, 1024, 23, 6),
    (0, 3072, 10, 6), (0, 3072, 13, 7), (1, 1536, 10, 6), (1, 1536, 13, 7), (1, 1536, 15, 6), (1, 1536, 17, 4), (1, 1536, 27, 7), (1, 2560, 9, 4), (1, 2560, 15, 4),   # two blocks of eight do not fit
    (0, 3840, 24, 8), (1, 1280, 20, 8),                                                                                 # an odd number of super-blocks
])
def test_warps_of_a_streamed_matvec(ctx, gate_up, cols, per_sm, warps):
    """One token without a plan takes the block size that was measured fastest for its groups per SM (on 148 SMs; see stream_q4k_warps)."""
    rows = int(per_sm * ctx.lib.ks_ctx_sm_count(ctx.h)) * (8 if cols // 256 % 2 else 4)
    bw, bx, y = (ctx.buffer_empty_bytes(n) for n in (rows * cols // 256 * 144, 4 * cols, 4 * rows))

    def call():
        if gate_up:
            ctx.check(ctx.lib.ks_matvec_gate_up_gelu(ctx.h, rows, cols, Q4K, bw.h, bw.h, 0, bx.h, y.h))
        else:
            ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, Q4K, bw.h, 0, 0, bx.h, 0, y.h, 0, 1))

    assert _blocks_of(ctx, call)[1] == 32 * warps


def test_few_rows_never_allocate_and_graphs_outlive_growth(oracle):
    """2..8 rows work out of the scratch the context starts with: device memory in use does not change, and a shape that would
    need more takes the matvec.  A graph captured over the scratch still gives its results after a larger batch has grown it."""
    import torch
    c = CudaContext(0)
    rows, cols = 2048, 1536
    W, x = _gen(Q4K, 74, "W", rows, cols), synth.normals(74, "x", 16 * cols).reshape(16, cols).astype(np.float32)
    y32, y64 = oracle.matvec(Q4K, W, rows, cols, x)
    bw, bx, y, y2 = c.buffer_bytes(W), c.buffer_bytes(x), c.buffer_empty_f32(16 * rows), c.buffer_empty_f32(16 * rows)
    most = 1 << 20                                            # rows: 8 x 2^20 sums are 32 MB by themselves
    big, bigx, bigy = c.buffer_empty_f32(most * 72), c.buffer_empty_f32(256 * 512), c.buffer_empty_f32(256 * (most // 4))
    c.synchronize()

    def call(r, k, bW, bX, bY, n):
        before = c.launch_count()
        c.check(c.lib.ks_matvec(c.h, r, k, Q4K, bW.h, 0, 0, bX.h, 0, bY.h, 0, n))
        return c.launch_count() - before

    call(rows, cols, bw, bx, y, 8)                            # the driver loads kernels on their first use
    call(most, 512, big, bigx, bigy, 8)
    c.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert call(rows, cols, bw, bx, y, 8) > 1                 # the GEMM
    _check(c.read_f32(y, 8 * rows).reshape(8, rows), y32[:8], y64[:8], "8 rows")
    assert call(most // 2, 512, big, bigx, bigy, 8) > 1 and call(most, 512, big, bigx, bigy, 8) == 1
    c.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    call(rows, cols, bw, bx, y, 16)
    c.check(c.lib.ks_graph_begin(c.h))
    c.check(c.lib.ks_matvec(c.h, rows, cols, Q4K, bw.h, 0, 0, bx.h, 0, y2.h, 0, 16))
    g = c.lib.ks_graph_end(c.h)
    assert g
    call(most // 4, 512, big, bigx, bigy, 256)
    c.synchronize()
    assert torch.cuda.mem_get_info()[0] < free - (200 << 20)  # the scratch has grown
    c.check(c.lib.ks_graph_launch(c.h, g))
    _check(c.read_f32(y2, 16 * rows).reshape(16, rows), y32, y64, "graph after growth")
    c.lib.ks_graph_free(c.h, g)
    c.close()


@pytest.mark.parametrize("dtype,rows,cols,batch,launches", [
    (Q4K, 4096, 1536, 3, (2, 3)), (Q4K, 1024, 10240, 4, (2, 3)), (Q4K, 16384, 512, 8, (2, 3)),   # the few-row kernels
    (Q4K, 1536, 1536, 3, (1,)), (Q4K, 2048, 1536, 3, (2, 3)), (Q4K, 1536, 1536, 4, (2, 3)),      # either side of the line for 3 rows
    (Q6K, 4096, 1536, 3, (2,)), (Q6K, 2048, 2560, 8, (2,)),
    (Q6K, 2048, 10240, 4, (1,)), (Q6K, 2007, 2048, 8, (1,)), (Q6K, 2056, 2048, 3, (1,)),         # outside the Q6_K one: the matvec
    (Q6K, 512, 10240, 8, (2, 3)),                                                                # more than the matvec can stage
])
def test_few_rows_are_as_exact_as_the_matvec(ctx, oracle, dtype, rows, cols, batch, launches):
    """2..8 token rows with a few channels a thousand times the rest, as activations have them, against 64 bits.  The batch
    matvec is 1.5e-7 off (relative 2-norm): f32 operands and sums of up to 10240 terms in 32-term blocks, a few 2^-24.  The
    bound is 3.5e-7, six units of 2^-24; sums that lose low bits against the large channels are ten times that."""
    W = _gen(dtype, 75, f"W{rows}x{cols}", rows, cols)
    x = synth.normals(75, f"x{cols}", batch * cols).reshape(batch, cols).astype(np.float32)
    x[:, 7::251] *= 1000.0
    off = 2 if (dtype, rows) == (Q6K, 2056) else 0
    bw = ctx.buffer_bytes(np.concatenate([np.zeros(off, np.uint8), np.frombuffer(W, np.uint8)]))
    bx, y = ctx.buffer_bytes(x), ctx.buffer_empty_f32(batch * rows)
    before = ctx.launch_count()
    ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, dtype, bw.h, off, 0, bx.h, 0, y.h, 0, batch))
    assert ctx.launch_count() - before in launches
    got = ctx.read_f32(y, batch * rows).reshape(batch, rows).astype(np.float64)
    want = x.astype(np.float64) @ oracle.dequant(dtype, W, rows * cols).astype(np.float64).reshape(rows, cols).T
    err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() <= (3.5e-7 if (dtype, cols, batch) != (Q6K, 10240, 8) else 1e-5), err   # there the tcgen05 kernel: f32 sums over all columns


@pytest.mark.parametrize("batch", [5, 24, 100])
def test_a_large_dmin_without_minima_changes_nothing(ctx, oracle, batch):
    """Super-blocks whose minima are all 0 with dmin 2^26 times d: the weights are d sc q, as with dmin = 0."""
    rows, cols = 130, 512
    W = np.frombuffer(_gen(Q4K, 77, "W", rows, cols), np.uint8).reshape(rows, cols // 256, 144).copy()
    sc = np.random.default_rng(77).integers(0, 64, (rows, cols // 256, 8), np.uint8)
    W[:, :, 4:8], W[:, :, 8:12] = (sc[:, :, :4] & 63) | ((sc[:, :, 4:] >> 4) << 6), 0
    W[:, :, 12:16] = sc[:, :, 4:] & 15
    W[0::2, :, 0:4] = np.frombuffer(np.array([2.0 ** -20, 64.0], np.float16).tobytes(), np.uint8)
    W[1::2, :, 0:4] = np.frombuffer(np.array([2.0 ** -20, 2.0 ** -3], np.float16).tobytes(), np.uint8)
    x = synth.normals(77, f"x{batch}", batch * cols).reshape(batch, cols).astype(np.float32)
    raw = W.tobytes()
    bw, bx, y = ctx.buffer_bytes(np.frombuffer(raw, np.uint8)), ctx.buffer_bytes(x), ctx.buffer_empty_f32(batch * rows)
    ctx.check(ctx.lib.ks_matvec(ctx.h, rows, cols, Q4K, bw.h, 0, 0, bx.h, 0, y.h, 0, batch))
    y32, y64 = oracle.matvec(Q4K, np.frombuffer(raw, np.uint8), rows, cols, x)
    _check(ctx.read_f32(y, batch * rows).reshape(batch, rows) * 2.0 ** 20, y32 * np.float32(2.0 ** 20), y64 * 2.0 ** 20, f"{batch} rows")


@pytest.mark.parametrize("batch", [1, 3, 9])
def test_weights_quantised_just_before(batch):
    """Weights written by the quantiser and read by the next op of the same stream, without a wait between (programmatic
    dependent launch on): the same bits as after a wait, every time."""
    rows, cols = 8192, 2560
    c = CudaContext(0, flags=1)
    rng = np.random.default_rng(76)
    w = [c.buffer_bytes(rng.standard_normal(rows * cols, np.float32)) for _ in range(2)]
    W, x = c.buffer_empty_bytes(rows * cols // 256 * 144), c.buffer_bytes(rng.standard_normal(batch * cols, np.float32))
    y = c.buffer_empty_f32(batch * rows)

    def run(i, wait):
        c.check(c.lib.ks_quantize_q4k(c.h, 0, w[i].h, 0, rows * cols, W.h, 0))
        if wait:
            c.synchronize()
        c.check(c.lib.ks_matvec(c.h, rows, cols, Q4K, W.h, 0, 0, x.h, 0, y.h, 0, batch))
        return c.read_f32(y, batch * rows)

    want = [run(i, True) for i in range(2)]
    for k in range(6):
        assert np.array_equal(run(k % 2, False), want[k % 2])
    c.close()
