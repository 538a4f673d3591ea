"""The streaming kernel on single CTAs (tcec_gemm_stream.cu): batches of matrices with at most 128 rows.

Against the FP64 oracle (tolerance: oracle.error_threshold, as in the other GEMM tests), and against the
same matrices one by one on CTA pairs, which form every sum in the same order."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T, Cj = api.CUBLAS_OP_N, api.CUBLAS_OP_T, api.CUBLAS_OP_C
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC
SCALING, AUTO = api.ComputeMode.FP16TCEC_SCALING, api.ComputeMode.AUTO


def _set(handle, value):
    if value is None:
        os.environ.pop("CUMPSGEMM_STREAM", None)
    else:
        os.environ["CUMPSGEMM_STREAM"] = str(value)
    handle.reload_tuning_env()


def _run(handle, oracle, cplx, op_a, op_b, m, n, k, mode, batch, beta):
    import torch

    q = 2 if cplx else 4                          # elements per 16 bytes
    up = lambda v: -(-v // q) * q                 # noqa: E731
    am, an = (m, k) if op_a == N else (k, m)
    bm, bn = (k, n) if op_b == N else (n, k)
    lda, ldb, ldc = up(am), up(bm), m + 1
    g = torch.Generator(device="cuda")
    g.manual_seed(m + 5 * n + 7 * k)

    def values(count):
        x = torch.rand((count, 2) if cplx else (count,), device="cuda", generator=g) * 2 - 1
        return torch.view_as_complex(x) if cplx else x

    a, b, c0 = values(lda * an * batch), values(ldb * bn * batch), values(ldc * n * batch)
    if beta == 0:
        c0.fill_(float("nan"))                    # must not be read
    alpha = 0.75 - 0.5j if cplx else 1.5
    out = []
    for value in (1, 128):                        # single CTAs, pairs
        c = c0.clone()
        _set(handle, value)
        try:
            handle.gemm_strided_batch(op_a, op_b, m, n, k, alpha, a, lda, lda * an, b, ldb, ldb * bn,
                                      beta, c, ldc, ldc * n, batch, mode)
            assert handle.last_route()[0] == api.ROUTE_STREAMING
            cut = handle.last_route()[1]
        finally:
            _set(handle, None)
        out.append(torch.view_as_real(c) if cplx else c)
    if not cut:                                   # (pieces of a tile are added in another order)
        assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32))
    ah, bh, ch, c0h = (t.cpu().numpy() for t in
                       (a, b, torch.view_as_complex(out[0]) if cplx else out[0], c0))
    for i in sorted({0, batch // 2, batch - 1}):
        truth = oracle.gemm_f64(op_a, op_b, m, n, k, alpha, ah[i * lda * an:], lda, bh[i * ldb * bn:],
                                ldb, beta, None if beta == 0 else c0h[i * ldc * n:], ldc)
        r = oracle.residual(truth, ch[i * ldc * n:(i + 1) * ldc * n], ldc)
        # (one product by itself may be off by the dropped lo * lo, 2^-22 of it, and by both los' rounding,
        # another 2^-22)
        assert r < max(oracle.error_threshold(True, k * (2 if cplx else 1)),
                       2.0 ** -21 if k == 1 else 0.0), (i, r)
    pad = ch.reshape(batch, n, ldc)[:, :, m]
    np.testing.assert_array_equal(pad, c0h.reshape(batch, n, ldc)[:, :, m])
    assert handle.kernel_status() == 0


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC, SCALING, AUTO])
@pytest.mark.parametrize("ops", [(N, N), (N, T), (T, N), (T, T)])
@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (128, 128, 64, 9), (127, 129, 65, 8), (64, 300, 200, 150),
                                   (100, 40, 97, 500)])
def test_real(handle, oracle, shape, ops, mode):
    m, n, k, batch = shape
    _run(handle, oracle, False, *ops, m, n, k, mode, batch, 0.0)
    _run(handle, oracle, False, *ops, m, n, k, mode, batch, 0.5)


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC, AUTO])
@pytest.mark.parametrize("ops", [(N, N), (N, Cj), (T, N), (Cj, T)])
@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (64, 128, 32, 9), (63, 65, 50, 300)])
def test_complex(handle, oracle, shape, ops, mode):
    m, n, k, batch = shape
    _run(handle, oracle, True, *ops, m, n, k, mode, batch, 0.5)
