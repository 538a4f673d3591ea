"""The kernel that splits its operands between TMA and the tensor core, forced on (width 256 and
128), against the FP64 oracle: every op and kind, edges of tiles and slots, K pieces, slices.

Tolerance: the pass criterion of the other GEMM tests (oracle.error_threshold)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T, Cj = api.CUBLAS_OP_N, api.CUBLAS_OP_T, api.CUBLAS_OP_C
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC
SCALING, AUTO = api.ComputeMode.FP16TCEC_SCALING, api.ComputeMode.AUTO


class _Stream:
    def __init__(self, handle, value):
        self.handle, self.value = handle, value

    def __enter__(self):
        os.environ["CUMPSGEMM_STREAM"] = str(self.value)
        self.handle.reload_tuning_env()

    def __exit__(self, *exc):
        os.environ.pop("CUMPSGEMM_STREAM", None)
        self.handle.reload_tuning_env()


def _gen(oracle, cplx, seed, count, scale=1.0):
    x = oracle.gen_uniform(seed, count)
    if cplx:
        x = (x + 1j * oracle.gen_uniform(seed + 1000, count)).astype(np.complex64)
    return (x * np.float32(scale)).astype(x.dtype)


def _check(handle, oracle, width, cplx, op_a, op_b, m, n, k, mode, batch=1, beta=0.0, scale=1.0,
           pad=0, shared_b=False, reps=1, cut=None):
    import torch

    q = 2 if cplx else 4                          # elements per 16 bytes
    up = lambda v: -(-v // q) * q + pad * q       # noqa: E731
    am, an = (m, k) if op_a == N else (k, m)
    bm, bn = (k, n) if op_b == N else (n, k)
    lda, ldb, ldc = up(am), up(bm), m + pad
    a = _gen(oracle, cplx, 1, lda * an * batch, scale)
    b = _gen(oracle, cplx, 2, ldb * bn * (1 if shared_b else batch), scale)
    c0 = _gen(oracle, cplx, 3, ldc * n * batch)
    if beta == 0:
        c0[:] = np.nan                            # must not be read
    alpha = 0.75 - 0.5j if cplx else 1.5
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    sb = 0 if shared_b else ldb * bn
    outs = []
    with _Stream(handle, width):
        for _ in range(reps):
            dc = torch.from_numpy(c0.copy()).cuda()
            handle.gemm_strided_batch(op_a, op_b, m, n, k, alpha, da, lda, lda * an, db, ldb, sb,
                                      beta, dc, ldc, ldc * n, batch, mode)
            route, was_cut = handle.last_route()
            assert route == api.ROUTE_STREAMING   # and not a route the call has fallen back to
            assert cut is None or was_cut == cut
            outs.append(dc.cpu().numpy())
    for o in outs[1:]:
        np.testing.assert_array_equal(o.view(np.uint32), outs[0].view(np.uint32))
    res = outs[0].reshape(batch, n, ldc)
    if pad:                                       # nothing outside the m rows is written
        np.testing.assert_array_equal(np.ascontiguousarray(res[:, :, m:]).view(np.uint32),
                                      np.ascontiguousarray(c0.reshape(res.shape)[:, :, m:]).view(np.uint32))
    for i in sorted({0, batch // 2, batch - 1}):
        truth = oracle.gemm_f64(op_a, op_b, m, n, k, alpha, a[i * lda * an:], lda,
                                b[0 if shared_b else i * ldb * bn:], ldb, beta,
                                None if beta == 0 else c0[i * ldc * n:], ldc)
        r = oracle.residual(truth, outs[0][i * ldc * n:(i + 1) * ldc * n], ldc)
        assert r < oracle.error_threshold(True, k * (2 if cplx else 1)), (i, r)


@pytest.mark.parametrize("width", [256, 128])
@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
@pytest.mark.parametrize("op_a,op_b", [(N, N), (N, T), (T, N), (T, T)])
def test_real_layouts(handle, oracle, width, mode, op_a, op_b):
    # one row, column and k value past the edges of a tile and of a slot
    _check(handle, oracle, width, False, op_a, op_b, 257, 129, 97, mode, beta=0.5, pad=1)


@pytest.mark.parametrize("width", [256, 128])
@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
@pytest.mark.parametrize("op_a", [N, T, Cj])
@pytest.mark.parametrize("op_b", [N, T, Cj])
def test_complex_layouts(handle, oracle, width, mode, op_a, op_b):
    _check(handle, oracle, width, True, op_a, op_b, 129, 130, 49, mode, batch=2, beta=0.5, pad=1)


@pytest.mark.parametrize("width", [256, 128])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 300, 5), (300, 1, 64), (256, 256, 32), (255, 257, 65)])
def test_smallest_and_edge_sizes(handle, oracle, width, shape):
    _check(handle, oracle, width, False, N, N, *shape, FP16TCEC)


@pytest.mark.parametrize("width", [256, 128])
@pytest.mark.parametrize("shape,batch,cut", [
    ((256, 256, 4096), 1, {256: True, 128: True}),     # slices, added by the piece kernel
    ((520, 300, 1500), 13, {256: True, 128: True}),    # pieces that end inside tiles
    ((520, 300, 1500), 10, {256: False, 128: True}),   # 60 (too many left over) and 90 tiles
    ((256, 250, 192), 76, {256: False, 128: False})])  # a whole wave plus a few tiles too short to cut
@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
def test_k_pieces_and_slices(handle, oracle, width, shape, batch, cut, mode):
    """Cut tiles: right, and bit-identical from run to run."""
    _check(handle, oracle, width, False, T, N, *shape, mode, batch=batch, beta=-0.5, reps=3,
           cut=cut[width])


@pytest.mark.parametrize("cplx,op_a,op_b", [(False, N, N), (False, T, T), (True, N, N), (True, Cj, T)])
@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
def test_interleaved_batches_have_the_bits_of_contiguous_ones(handle, oracle, cplx, op_a, op_b, mode):
    """Matrices of a batch interleaved column by column (batch stride = one column, leading dimension =
    batch columns), and overlapping ones (stride of one 16-byte group): the same bits as from copies
    laid out one behind the other."""
    import torch

    m, n, k, batch = 132, 72, 52, 12
    q = 2 if cplx else 4
    am, an = (m, k) if op_a == N else (k, m)
    bm, bn = (k, n) if op_b == N else (n, k)
    a = torch.from_numpy(_gen(oracle, cplx, 1, am * an * batch)).cuda()
    b = torch.from_numpy(_gen(oracle, cplx, 2, bm * bn * batch)).cuda()

    def run(da, lda, sa, db, ldb, sb):
        c = torch.zeros(batch * m * n, dtype=a.dtype, device="cuda")
        with _Stream(handle, 1):
            handle.gemm_strided_batch(op_a, op_b, m, n, k, 1.0, da, lda, sa, db, ldb, sb, 0.0, c, m, m * n,
                                      batch, mode)
        assert handle.last_route()[0] == api.ROUTE_STREAMING
        return c

    # the storage read as [column][batch][row], and copied to [batch][column][row]
    flat = lambda x, cols, rows: x.view(cols, batch, rows).permute(1, 0, 2).contiguous().view(-1)  # noqa: E731
    got = run(a, am * batch, am, b, bm * batch, bm)
    want = run(flat(a, an, am), am, am * an, flat(b, bn, bm), bm, bm * bn)
    assert torch.equal(got, want)
    # overlapping: matrix i starts q elements after matrix i - 1
    got = run(a, am, q, b, bm, q)
    shifted = lambda x, size: torch.cat([x[i * q:i * q + size] for i in range(batch)])             # noqa: E731
    want = run(shifted(a, am * an), am, am * an, shifted(b, bm * bn), bm, bm * bn)
    assert torch.equal(got, want)


@pytest.mark.parametrize("width", [256, 128])
def test_scaling_shared_operand_and_short_tiles(handle, oracle, width):
    """Scale factors reach both converters; a batch stride of zero shares one matrix; three waves
    of short tiles (the 128-wide kernel then stores from registers), complex alpha."""
    _check(handle, oracle, width, True, N, N, 130, 70, 60, SCALING, batch=24, scale=2.0 ** -22)
    _check(handle, oracle, width, False, N, T, 200, 100, 70, FP16TCEC, batch=16, shared_b=True)
    _check(handle, oracle, width, True, N, N, 128, 100, 64, FP16TCEC, batch=240)
    _check(handle, oracle, width, False, N, N, 250, 120, 128, TF32TCEC, batch=240)


@pytest.mark.parametrize("wide", [False, True])
def test_auto_decides_on_the_device(handle, oracle, wide):
    """One launch reads the decision and runs the FP16 or the TF32 pipeline."""
    import torch

    m, n, k = 200, 260, 300
    a, b = oracle.gen_uniform(1, m * k), oracle.gen_uniform(2, k * n)
    if wide:
        a = np.ldexp(a, np.random.default_rng(0).integers(-30, 10, a.size)).astype(np.float32)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    dc = torch.zeros(m * n, device="cuda")
    with _Stream(handle, 1):
        ia, ib = handle.exp_stats_ext(m, k, da, m), handle.exp_stats_ext(k, n, db, k)
        handle.gemm_strided_batch_with_stats(N, N, m, n, k, 1.0, da, m, 0, db, k, 0, 0.0, dc, m, 0, 1,
                                             AUTO, ia, ib)
        assert handle.last_route()[0] == api.ROUTE_STREAMING
    if wide:
        assert handle.get_exp_stats_compute_mode_level(ia) == TF32TCEC
    truth = oracle.gemm_f64(N, N, m, n, k, 1.0, a, m, b, k, 0.0, None, m)
    assert oracle.residual(truth, dc.cpu().numpy(), m) < oracle.error_threshold(True, k)


def test_calls_tma_cannot_address_take_another_path(handle, oracle):
    """Unaligned leading dimension or base: refused by the rule, computed all the same."""
    import torch

    m, n, k = 130, 90, 77
    a, b = oracle.gen_uniform(1, (m + 1) * k + 1), oracle.gen_uniform(2, (k + 3) * n)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    truth = oracle.gemm_f64(N, N, m, n, k, 1.0, a, m + 1, b, k + 3, 0.0, None, m)
    off = oracle.gemm_f64(N, N, 128, n, 64, 1.0, a[1:], 128, b, k + 3, 0.0, None, 128)
    with _Stream(handle, 1):
        c = torch.zeros(m * n, device="cuda")
        handle.gemm(N, N, m, n, k, 1.0, da, m + 1, db, k + 3, 0.0, c, m, FP16TCEC)
        assert handle.last_route()[0] == api.ROUTE_PRESPLIT_SINGLE
        assert oracle.residual(truth, c.cpu().numpy(), m) < oracle.error_threshold(True, k)
        c = torch.zeros(128 * n, device="cuda")
        handle.gemm(N, N, 128, n, 64, 1.0, da[1:], 128, db, k + 3, 0.0, c, 128, TF32TCEC)
        assert handle.last_route()[0] == api.ROUTE_PRESPLIT_SINGLE
        assert oracle.residual(off, c.cpu().numpy(), 128) < oracle.error_threshold(True, 64)
