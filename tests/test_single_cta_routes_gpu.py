"""The streaming kernel on single CTAs and the kernel for small products: that they ran (Handle.last_tile),
infinities and NaN, leading dimensions beyond the smallest, operands shared by a whole batch.

A finite result is compared with the FP64 oracle (tolerance: oracle.error_threshold, as in the other GEMM
tests).  A non-finite element of A spoils its row of C, one of B its column (lo of an infinity is NaN); all
else keeps its bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T = api.CUBLAS_OP_N, api.CUBLAS_OP_T
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC
SOLO = (api.ROUTE_STREAMING, (128, 128))
SMALL = (api.ROUTE_ON_THE_FLY, (128, 32))


def _ran(handle):
    return handle.last_route()[0], handle.last_tile()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("kernel,m,n,k,batch", [
    (SOLO, 100, 300, 128, 240), (SOLO, 100, 60, 96, 700),          # looped stores / straight from registers
    (SMALL, 150, 70, 64, 2), (SMALL, 96, 33, 50, 1)])
@pytest.mark.parametrize("mode,op_a", [(FP16TCEC, N), (TF32TCEC, T)])
def test_a_non_finite_operand_reaches_its_row_and_column_only(handle, oracle, kernel, m, n, k, batch, value,
                                                              mode, op_a):
    import torch

    a, b = oracle.gen_uniform(1, batch * m * k), oracle.gen_uniform(2, batch * k * n)
    lda = m if op_a == N else k
    i, j = batch - 1, 0                           # matrices of the batch that are hit
    row, col, ka, kb = m - 1, n - 1, k - 1, 3
    bad_a, bad_b = a.copy(), b.copy()
    bad_a[i * m * k + (row + ka * lda if op_a == N else ka + row * lda)] = value
    bad_b[j * k * n + kb + col * k] = value
    outs = []
    for x, y in ((bad_a, bad_b), (a, b)):
        da, db = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        c = torch.full((batch * m * n,), float("nan"), device="cuda")
        handle.gemm_strided_batch(op_a, N, m, n, k, 1.0, da, lda, m * k, db, k, k * n, 0.0, c, m, m * n,
                                  batch, mode)
        assert _ran(handle) == kernel
        outs.append(c.cpu().numpy().reshape(batch, n, m))
    got, clean = outs
    assert np.isfinite(clean).all()
    hit = np.zeros((batch, n, m), bool)
    hit[i, :, row] = True
    hit[j, col, :] = True
    assert np.isnan(got[hit]).all()
    np.testing.assert_array_equal(got[~hit].view(np.uint32), clean[~hit].view(np.uint32))


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
@pytest.mark.parametrize("shared", ["", "a", "b"])
@pytest.mark.parametrize("op_a,op_b", [(N, N), (T, N), (N, T)])
def test_solo_with_wide_leading_dimensions_and_shared_operands(handle, oracle, mode, shared, op_a, op_b):
    """What lies between the columns, and beyond a matrix, is NaN: it must not be read into a result."""
    import torch

    m, n, k, batch = 90, 130, 70, 400
    am, an = (m, k) if op_a == N else (k, m)
    bm, bn = (k, n) if op_b == N else (n, k)
    lda, ldb, ldc = am + 10 + (-am - 10) % 4, bm + 20 + (-bm - 20) % 4, m + 7
    sa, sb = (0 if shared == "a" else lda * an + 8), (0 if shared == "b" else ldb * bn + 4)

    def operand(seed, rows, cols, ld, stride):
        x = np.full((1 if stride == 0 else batch, stride or ld * cols), np.nan, np.float32)
        v = oracle.gen_uniform(seed, x.shape[0] * rows * cols).reshape(x.shape[0], cols, rows)
        x[:, :ld * cols].reshape(x.shape[0], cols, ld)[:, :, :rows] = v
        return x

    a, b = operand(3, am, an, lda, sa), operand(4, bm, bn, ldb, sb)
    c = torch.full((batch * ldc * n,), -7.0, device="cuda")
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    handle.gemm_strided_batch(op_a, op_b, m, n, k, 1.0, da, lda, sa, db, ldb, sb, 0.0, c, ldc, ldc * n, batch,
                              mode)
    assert _ran(handle) == SOLO
    ch = c.cpu().numpy()
    for i in (0, batch // 3, batch - 1):
        truth = oracle.gemm_f64(op_a, op_b, m, n, k, 1.0, a[i if sa else 0], lda, b[i if sb else 0], ldb, 0.0,
                                None, ldc)
        assert oracle.residual(truth, ch[i * ldc * n:(i + 1) * ldc * n], ldc) < oracle.error_threshold(True, k)
    assert (ch.reshape(batch, n, ldc)[:, :, m:] == -7.0).all()
    assert handle.kernel_status() == 0


@pytest.mark.parametrize("m,n,k,batch", [(128, 128, 64, 9), (127, 129, 65, 64), (64, 300, 200, 150),
                                         (100, 40, 97, 500)])
def test_the_switch_selects_single_ctas(handle, monkeypatch, m, n, k, batch):
    """CUMPSGEMM_STREAM=1 against 128 is the comparison of another test: here, that they differ."""
    import torch

    lda, ldb = -(-m // 4) * 4, -(-k // 4) * 4
    a, b, c = (torch.zeros(x * batch, device="cuda") for x in (lda * k, ldb * n, m * n))
    for value, tile in ((1, (128, 128)), (128, (256, 128)), (256, (256, 256))):
        monkeypatch.setenv("CUMPSGEMM_STREAM", str(value))
        handle.reload_tuning_env()
        handle.gemm_strided_batch(N, N, m, n, k, 1.0, a, lda, lda * k, b, ldb, ldb * n, 0.0, c, m, m * n,
                                  batch, FP16TCEC)
        assert _ran(handle) == (api.ROUTE_STREAMING, tile)
    monkeypatch.delenv("CUMPSGEMM_STREAM")
    handle.reload_tuning_env()
