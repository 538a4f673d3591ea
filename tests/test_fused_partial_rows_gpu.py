"""The kernel that splits on the fly (CUMPSGEMM_FUSED=1) where a warp holds the last rows of a complex
matrix and some beyond it, C is not read and alpha is real: both ways to store apply to the warp's lanes.
Against the FP64 oracle (tolerance: oracle.error_threshold, as in the other GEMM tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N = api.CUBLAS_OP_N


@pytest.mark.parametrize("m,n,k,batch", [(36, 128, 64, 8), (2, 912, 512, 20), (64, 64, 32, 8), (70, 130, 96, 9)])
def test_complex_with_a_real_alpha(handle, oracle, monkeypatch, m, n, k, batch):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(m + n)
    values = lambda c: torch.view_as_complex(torch.rand((c, 2), device="cuda", generator=g) * 2 - 1)  # noqa: E731
    a, b = values(batch * m * k), values(batch * k * n)
    c = torch.full((batch * m * n,), complex("nan"), device="cuda", dtype=torch.complex64)
    monkeypatch.setenv("CUMPSGEMM_FUSED", "1")
    handle.reload_tuning_env()
    try:
        handle.gemm_strided_batch(N, N, m, n, k, 1.5, a, m, m * k, b, k, k * n, 0.0, c, m, m * n, batch,
                                  api.ComputeMode.FP16TCEC)
        assert handle.last_route()[0] == api.ROUTE_ON_THE_FLY
    finally:
        monkeypatch.delenv("CUMPSGEMM_FUSED")
        handle.reload_tuning_env()
    ah, bh, ch = (t.cpu().numpy() for t in (a, b, c))
    for i in sorted({0, batch - 1}):
        truth = oracle.gemm_f64(N, N, m, n, k, 1.5, ah[i * m * k:], m, bh[i * k * n:], k, 0.0, None, m)
        assert oracle.residual(truth, ch[i * m * n:(i + 1) * m * n], m) < oracle.error_threshold(True, 2 * k)
    assert handle.kernel_status() == 0
