"""cuMpSGEMM_sgemm_static_scratch on sizes that fit its 32 MiB array only with a narrower tile than
the fastest one: they are computed, not refused (a caller without a way to allocate has no other
entry point), against the FP64 oracle with the suite's pass criterion."""
import os

import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

FP16TCEC, TF32TCEC = 1, 2


def _panel_bytes(mode, m, n, k, tile_m, tile_n):
    up = lambda v, q: -(-v // q) * q              # noqa: E731
    return (4 if mode == FP16TCEC else 8) * (up(m, tile_m) + up(n, tile_n)) * up(k, 64)


@pytest.mark.parametrize("mode,m,n,k", [
    (FP16TCEC, 1034, 2153, 2483),    # 256 columns need 34.5 MB, 128 columns 33.2
    (FP16TCEC, 512, 2496, 2752),     # 128 columns need 33.8 MB, 64 columns 33.1
    (FP16TCEC, 1202, 901, 3683),
    (TF32TCEC, 2944, 832, 1088),
])
def test_narrower_tile_where_the_fastest_does_not_fit(oracle, mode, m, n, k):
    import torch

    assert _panel_bytes(mode, m, n, k, 128, 64) <= 32 << 20
    assert _panel_bytes(mode, m, n, k, 256, 256) > 32 << 20
    a, b, c0 = oracle.gen_uniform(1, m * k), oracle.gen_uniform(2, k * n), oracle.gen_uniform(3, m * n)
    da, db, dc = (torch.from_numpy(x.copy()).cuda() for x in (a, b, c0))
    stream = torch.cuda.current_stream()
    st = api.sgemm_static_scratch(stream, 0, 0, m, n, k, 1.0, da, m, db, k, 0.5, dc, m, mode)
    assert st == api.CUBLAS_STATUS_SUCCESS
    truth = oracle.gemm_f64(0, 0, m, n, k, 1.0, a, m, b, k, 0.5, c0, m)
    assert oracle.residual(truth, dc.cpu().numpy(), m) < oracle.error_threshold(True, k)
    # a tile the caller forces is kept: refused when its panels do not fit
    os.environ["CUMPSGEMM_TILE_N"] = "256"
    try:
        st = api.sgemm_static_scratch(stream, 0, 0, m, n, k, 1.0, da, m, db, k, 0.5, dc, m, mode)
        assert st == api.CUBLAS_STATUS_INVALID_VALUE
    finally:
        os.environ.pop("CUMPSGEMM_TILE_N", None)
