"""The one-launch kernel for small products (tcec_gemm_small.cu) against the pre-split path.

Both feed the tensor core the same hi / lo bits, chunk by chunk, and add in the same order, so the results
are equal bit for bit; CUMPSGEMM_TILE_N=64 forces the pre-split path."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T, Cj = api.CUBLAS_OP_N, api.CUBLAS_OP_T, api.CUBLAS_OP_C
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC
SCALING, AUTO = api.ComputeMode.FP16TCEC_SCALING, api.ComputeMode.AUTO

# one row / column / k value, remainders of the 128 x 32 tile and of a chunk (64 / 32 k values), and on
# both sides of the rule's two limits: 2 and 4 chunks
SHAPES = [(1, 1, 1), (128, 32, 64), (129, 33, 65), (300, 17, 31), (5, 100, 127), (257, 95, 200),
          (128, 128, 128), (40, 50, 256), (40, 50, 257)]


def _one_launch(cplx, m, n, k, mode, batch):
    """The rule of gemm_api.cu for products of at most 148 tiles."""
    q = 2 if cplx else 1
    chunks = -(-k * q // (32 if mode in (TF32TCEC, AUTO) else 64))
    assert -(-m * q // 128) * -(-n // 32) * batch <= 148
    return chunks <= (2 if mode in (SCALING, AUTO) else 4)


def _forced(handle, on):
    if on:
        os.environ["CUMPSGEMM_TILE_N"] = "64"
    else:
        os.environ.pop("CUMPSGEMM_TILE_N", None)
    handle.reload_tuning_env()


def _both(handle, cplx, op_a, op_b, m, n, k, mode, batch, pad, beta, offset=0, nan_tail=False):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(m * 7 + n * 3 + k)
    dt = torch.complex64 if cplx else torch.float32
    am, an = (m, k) if op_a == N else (k, m)
    bm, bn = (k, n) if op_b == N else (n, k)
    lda, ldb, ldc = am + pad, bm + pad, m + pad

    def values(count):
        x = torch.randn((count, 2) if cplx else (count,), device="cuda", generator=g)
        return torch.view_as_complex(x) if cplx else x

    a, b = values(lda * an * batch + offset)[offset:], values(ldb * bn * batch + offset)[offset:]
    if nan_tail and pad:  # what lies between the columns is not part of the operand
        a.view(-1)[: lda * an * batch].reshape(batch, an, lda)[:, :, am:] = float("nan")
        b.view(-1)[: ldb * bn * batch].reshape(batch, bn, ldb)[:, :, bm:] = float("nan")
    c0 = values(ldc * n * batch) if beta != 0 else torch.full((ldc * n * batch,), float("nan"),
                                                              device="cuda", dtype=dt)
    alpha = 0.75 - 0.5j if cplx else 1.5
    out = []
    for forced in (False, True):
        c = c0.clone()
        _forced(handle, forced)
        try:
            handle.gemm_strided_batch(op_a, op_b, m, n, k, alpha, a, lda, lda * an, b, ldb, ldb * bn,
                                      beta, c, ldc, ldc * n, batch, mode)
            route = handle.last_route()[0]
        finally:
            _forced(handle, False)
        if forced or _one_launch(cplx, m, n, k, mode, batch):
            assert route == (api.ROUTE_PRESPLIT_SINGLE if forced else api.ROUTE_ON_THE_FLY)
        else:
            assert route != api.ROUTE_ON_THE_FLY
        out.append(torch.view_as_real(c) if cplx else c)
    assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32))
    valid = out[0].reshape(batch, n, ldc, -1)[:, :, :m]
    assert torch.isfinite(valid).all()
    if pad and beta == 0:
        assert torch.isnan(out[0].reshape(batch, n, ldc, -1)[:, :, m:]).all()
    assert handle.kernel_status() == 0
    return a, b, c0, lda, ldb, ldc, out[0]


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC, SCALING, AUTO])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("ops", [(N, N), (N, T), (T, N), (T, T)])
def test_real_equals_presplit(handle, ops, shape, mode):
    _both(handle, False, *ops, *shape, mode, batch=2, pad=1, beta=0.5)
    _both(handle, False, *ops, *shape, mode, batch=1, pad=0, beta=0.0)


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC, SCALING, AUTO])
@pytest.mark.parametrize("shape", [(1, 1, 1), (64, 32, 32), (65, 33, 33), (130, 40, 100)])
@pytest.mark.parametrize("ops", [(N, N), (N, Cj), (T, N), (Cj, T), (Cj, Cj)])
def test_complex_equals_presplit(handle, ops, shape, mode):
    _both(handle, True, *ops, *shape, mode, batch=2, pad=3, beta=0.5)
    _both(handle, True, *ops, *shape, mode, batch=1, pad=0, beta=0.0)


@pytest.mark.parametrize("ops", [(N, N), (T, T)])
def test_unaligned_base_and_poisoned_padding(handle, ops):
    """A base four bytes off, and NaN between the columns of the operands."""
    _both(handle, False, *ops, 130, 50, 170, FP16TCEC, batch=1, pad=0, beta=0.0, offset=1)
    _both(handle, False, *ops, 130, 50, 170, FP16TCEC, batch=2, pad=2, beta=0.5, nan_tail=True)


def test_against_the_oracle(handle, oracle):
    m, n, k = 129, 33, 65
    a, b, c0, lda, ldb, ldc, out = _both(handle, False, T, N, m, n, k, FP16TCEC, 1, 0, 0.5)
    truth = oracle.gemm_f64(T, N, m, n, k, 1.5, a.cpu().numpy(), lda, b.cpu().numpy(), ldb, 0.5,
                            c0.cpu().numpy(), ldc)
    assert oracle.residual(truth, out.cpu().numpy(), ldc) < oracle.error_threshold(True, k)
