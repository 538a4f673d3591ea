"""Sums that few products make up, on the kernel that splits its operands on the way: the corrections
must not cost hi*hi any bits.  One non-zero per row of A, so every element of C is one product.

Bounds.  hi holds 11 bits and lo 11 more, so a value differs from hi + lo by at most 2^-23 of itself; the
product leaves out lo * lo, at most 2^-22 of it; the sum of hi*hi and the corrections is rounded once
(2^-24): 2 * 2^-23 + 2^-22 + 2^-24.  All of these errors have either sign, so their mean over C is 0 up to
chance.  An element of A is shared by a row of C, so chance is largest in its share: errors
spread over +-2^-23 have a deviation of 2^-23 / sqrt(3), their mean over the rows a sqrt(rows)-th of it;
five times that.  A truncation of the finished sums shifts the mean by about 2^-25."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N = api.CUBLAS_OP_N
LARGEST = 2.0 ** -21 + 2.0 ** -24


def _errors(handle, width, mode, m, n, k, batch, small_b):
    """Relative errors of all elements of C."""
    import torch

    rng = np.random.default_rng(k)
    a = np.zeros((batch, k, m), np.float32)       # column-major: m runs fastest
    at = rng.integers(0, k, (batch, m))
    for i in range(batch):
        a[i, at[i], np.arange(m)] = 1 + rng.random(m)
    if small_b:                                   # exact in FP16 below 2^-13, subnormal below 2^-14
        b = np.ldexp(rng.integers(1, 1 << 13, (batch, n, k)), -23)
    else:
        b = 1 + rng.random((batch, n, k))
    b = (b * rng.choice([-1.0, 1.0], b.shape)).astype(np.float32)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    dc = torch.zeros((batch, n, m), dtype=torch.float32, device="cuda")
    os.environ["CUMPSGEMM_STREAM"] = str(width)
    handle.reload_tuning_env()
    try:
        handle.gemm_strided_batch(N, N, m, n, k, 1.0, da, m, m * k, db, k, k * n, 0.0, dc, m, m * n,
                                  batch, mode)
        assert handle.last_route()[0] == api.ROUTE_STREAMING
        c = dc.cpu().numpy().astype(np.float64)
    finally:
        os.environ.pop("CUMPSGEMM_STREAM")
        handle.reload_tuning_env()
    truth = b.astype(np.float64) @ a.astype(np.float64)
    return c / truth - 1


@pytest.mark.parametrize("mode", [api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC])
@pytest.mark.parametrize("width,m,n,k,batch", [
    (256, 512, 512, 68, 1), (256, 512, 512, 1024, 1), (128, 512, 512, 68, 1), (128, 512, 512, 1024, 1),
    (1, 128, 128, 256, 64),                       # (single CTAs: batches of at most 128 rows)
])
@pytest.mark.parametrize("small_b", [False, True])
def test_corrections_cost_no_bits_of_the_main_product(handle, mode, width, m, n, k, batch, small_b):
    e = _errors(handle, width, mode, m, n, k, batch, small_b)
    assert np.abs(e).max() <= LARGEST
    assert abs(e.mean()) <= 5 * 2.0 ** -23 / np.sqrt(3 * m * batch)
