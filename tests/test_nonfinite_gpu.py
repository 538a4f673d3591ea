"""Infinities and NaN through the GEMM kernels: what a non-finite operand or an overflowing sum
reaches, and what it does not, on the streaming kernel, the pre-split kernels (rolled epilogue) and
the kernel that adds K pieces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T = api.CUBLAS_OP_N, api.CUBLAS_OP_T
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC


def _set(handle, monkeypatch, **switches):
    for name in ("STREAM", "PAIR", "TILE_N", "SPLIT_K", "TAIL_SPLIT"):
        monkeypatch.delenv("CUMPSGEMM_" + name, raising=False)
    for name, value in switches.items():
        monkeypatch.setenv("CUMPSGEMM_" + name, str(value))
    handle.reload_tuning_env()


def test_an_infinite_sum_of_a_complex_product_is_the_same_on_every_path(handle, monkeypatch):
    """2^100 x 2^100 summed overflows FP32 in the real part only (powers of two: lo is zero, so no
    other term is involved).  With a real alpha the complex product still multiplies the infinity by
    alpha's zero imaginary part: the imaginary part is NaN, on whichever path."""
    import torch

    batch, m, n, k = 240, 128, 100, 64
    big = 2.0 ** 100
    a = torch.zeros(batch * m * k, dtype=torch.complex64, device="cuda")
    b = torch.zeros(batch * k * n, dtype=torch.complex64, device="cuda")
    a.view(batch, k, m)[:, :, 5] = big            # row 5 of every op(A)
    b.view(batch, n, k)[:, 7, :] = big            # column 7 of every op(B)
    results = []
    for switches in ({"STREAM": 128}, {"STREAM": 256}, {"STREAM": 0, "PAIR": 1},
                     {"STREAM": 0, "PAIR": 0, "TILE_N": 64}):
        _set(handle, monkeypatch, **switches)
        c = torch.zeros(batch * m * n, dtype=torch.complex64, device="cuda")
        handle.gemm_strided_batch(N, N, m, n, k, 1.5, a, m, m * k, b, k, k * n, 0.0, c, m, m * n, batch,
                                  TF32TCEC)
        results.append(c.cpu().numpy().reshape(batch, n, m))
    _set(handle, monkeypatch)
    want = np.zeros((batch, n, m), np.complex64)
    want[:, 7, 5] = complex(np.inf, np.nan)
    for c in results:
        np.testing.assert_array_equal(c.real, want.real)
        np.testing.assert_array_equal(c.imag, want.imag)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("switches,batch", [
    ({"STREAM": 256}, 1), ({"STREAM": 128}, 1),   # few tiles: K pieces, added by a second kernel
    ({"STREAM": 256, "TAIL_SPLIT": 0, "SPLIT_K": 0}, 1),
    ({"STREAM": 128}, 240),                       # stores straight from registers
    ({"STREAM": 0, "PAIR": 1}, 1), ({"STREAM": 0, "PAIR": 1, "TAIL_SPLIT": 0}, 1),
    ({"STREAM": 0, "PAIR": 0, "TILE_N": 128}, 1), ({"STREAM": 0, "PAIR": 0, "SPLIT_K": 4}, 1)])
@pytest.mark.parametrize("mode,op_a", [(FP16TCEC, N), (TF32TCEC, T)])
def test_a_non_finite_operand_reaches_its_row_and_column_only(handle, oracle, monkeypatch, switches, batch,
                                                              value, mode, op_a):
    """One non-finite element of A spoils its row of C, one of B its column (lo of an infinity is
    NaN, so the error-corrected product is NaN there); everything else is the finite result; C is not
    read with beta = 0."""
    import torch

    m, n, k = (200, 100, 128) if batch > 1 else (300, 200, 4096)
    lda = m if op_a == N else k
    a, b = oracle.gen_uniform(1, batch * m * k), oracle.gen_uniform(2, batch * k * n)
    i, j = batch - 1, 0                           # matrices of the batch that are hit
    row, col, ka, kb = m - 1, n - 1, k - 1, 3
    clean_a, clean_b = a.copy(), b.copy()
    a[i * m * k + (row + ka * lda if op_a == N else ka + row * lda)] = value
    b[j * k * n + kb + col * k] = value
    outs = []
    _set(handle, monkeypatch, **switches)
    for x, y in ((a, b), (clean_a, clean_b)):
        da, db = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        c = torch.full((batch * m * n,), float("nan"), device="cuda")
        handle.gemm_strided_batch(op_a, N, m, n, k, 1.0, da, lda, m * k, db, k, k * n, 0.0, c, m, m * n,
                                  batch, mode)
        outs.append(c.cpu().numpy().reshape(batch, n, m))
    _set(handle, monkeypatch)
    got, clean = outs
    assert np.isfinite(clean).all()
    hit = np.zeros((batch, n, m), bool)
    hit[i, :, row] = True
    hit[j, col, :] = True
    assert np.isnan(got[hit]).all()
    np.testing.assert_array_equal(got[~hit].view(np.uint32), clean[~hit].view(np.uint32))
