"""Which path a call takes (Handle.last_route) at sizes where one is faster by a tenth or more: batches of few
small matrices, where single CTAs with a long K loop of their own are slower than the split pass and the
GEMM behind it (us, streaming / pre-split: 8 x 128 x 128 x 512 12.6 / 8.9 FP16TCEC, 18.6 / 12.6 TF32TCEC),
and batches of many, which stream.  The choice must not depend on the layouts another kernel knows."""
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T, Cj = api.CUBLAS_OP_N, api.CUBLAS_OP_T, api.CUBLAS_OP_C
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC
PRESPLIT = (api.ROUTE_PRESPLIT_SINGLE, api.ROUTE_PRESPLIT_PAIR)


def _route(handle, cplx, op_a, op_b, m, n, k, batch, mode):
    import torch

    dt = torch.complex64 if cplx else torch.float32
    a, b, c = (torch.zeros(batch * x, dtype=dt, device="cuda") for x in (m * k, k * n, m * n))
    lda, ldb = (m if op_a == N else k), (k if op_b == N else n)
    handle.gemm_strided_batch(op_a, op_b, m, n, k, 1.0, a, lda, m * k, b, ldb, k * n, 0.0, c, m, m * n, batch,
                              mode)
    return handle.last_route()[0]


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
@pytest.mark.parametrize("cplx,ops", [(False, (N, N)), (False, (T, N)), (False, (N, T)), (False, (T, T)),
                                      (True, (N, N)), (True, (Cj, N)), (True, (T, T))])
def test_few_small_matrices(handle, cplx, ops, mode):
    m, k = (64, 256) if cplx else (128, 512)      # of the same real product
    assert _route(handle, cplx, *ops, m, 128, k, 8, mode) in PRESPLIT


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
@pytest.mark.parametrize("cplx,ops", [(False, (N, N)), (False, (T, T)), (True, (N, N)), (True, (Cj, N))])
@pytest.mark.parametrize("m,n,k,batch", [(64, 64, 96, 1000), (128, 128, 128, 1024), (256, 256, 256, 300),
                                         (32, 500, 44, 1500)])
def test_many_small_matrices(handle, cplx, ops, m, n, k, batch, mode):
    if cplx:
        m, k = m // 2, k // 2
    assert _route(handle, cplx, *ops, m, n, k, batch, mode) == api.ROUTE_STREAMING


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
@pytest.mark.parametrize("m,n,k,batch", [(128, 128, 512, 8), (700, 520, 700, 1)])
def test_a_call_without_memory_for_panels_streams(oracle, mode, m, n, k, batch):
    """A captured call on a handle without a workspace: pre-split by estimate, but streaming needs no memory."""
    import torch

    a, b = oracle.gen_uniform(1, batch * m * k), oracle.gen_uniform(2, batch * k * n)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    c = torch.zeros(batch * m * n, device="cuda")

    def call(h):
        h.gemm_strided_batch(N, N, m, n, k, 1.0, da, m, m * k, db, k, k * n, 0.0, c, m, m * n, batch, mode)
        return h.last_route()[0]

    with api.Handle() as h:                       # loads the kernels
        h.use_current_torch_stream()
        assert call(h) in PRESPLIT
        torch.cuda.synchronize()
    with api.Handle() as h:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            h.use_current_torch_stream()
            assert call(h) == api.ROUTE_STREAMING
        c.zero_()
        graph.replay()
        torch.cuda.synchronize()
        ch = c.cpu().numpy()
        for i in {0, batch - 1}:
            truth = oracle.gemm_f64(N, N, m, n, k, 1.0, a[i * m * k:], m, b[i * k * n:], k, 0.0, None, m)
            assert oracle.residual(truth, ch[i * m * n:(i + 1) * m * n], m) < oracle.error_threshold(True, k)
        del graph
        assert h.kernel_status() == 0
