"""The handle's workspace: who may free it, and when it may grow."""
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T = api.CUBLAS_OP_N, api.CUBLAS_OP_T
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC
SLACK = 4 << 20                                   # granularity of cudaMalloc


def _free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_a_graph_keeps_the_workspace_it_was_captured_with(oracle):
    """64 products of 512 x 512 x 1024 are 256 pair tiles; the 34 left over from the whole waves are
    cut along K and their sums go through the workspace.  A graph captured from such a call has to
    stay valid when a larger call makes the handle's workspace grow: the memory it writes to must not
    be given back.  (That is asserted on the free memory before the graph is replayed.)"""
    import torch

    batch, m, n, k = 64, 512, 512, 1024
    big = 4096
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    a = torch.rand(batch * m * k, device="cuda", generator=g) * 2 - 1
    b = torch.rand(batch * k * n, device="cuda", generator=g) * 2 - 1
    c = torch.zeros(batch * m * n, device="cuda")
    x, y = torch.ones(big * big, device="cuda"), torch.zeros(big * big, device="cuda")

    def small_call(h):
        h.use_current_torch_stream()
        h.gemm_strided_batch(N, N, m, n, k, 1.0, a, m, m * k, b, k, k * n, 0.0, c, m, m * n, batch,
                             FP16TCEC)

    def big_call(h):
        h.use_current_torch_stream()
        h.gemm(N, N, big, big, big, 1.0, x, big, x, big, 0.0, y, big, TF32TCEC)

    with api.Handle() as h:                       # loads the kernels
        small_call(h)
        big_call(h)
        torch.cuda.synchronize()
    with api.Handle() as h:                       # what the larger call takes by itself
        before = _free_bytes()
        big_call(h)
        alone = before - _free_bytes()
    with api.Handle() as h:                       # without a graph the outgrown block goes back
        before = _free_bytes()
        small_call(h)
        pieces = before - _free_bytes()
        assert 4 * SLACK < pieces < 64 << 20
        big_call(h)
        assert before - _free_bytes() <= alone + SLACK
    with api.Handle() as h:
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            small_call(h)
        side.synchronize()
        want = c.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            small_call(h)
        torch.cuda.synchronize()
        before = _free_bytes()
        big_call(h)
        assert before - _free_bytes() >= alone - SLACK
        c.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(c, want)
        del graph
        assert h.kernel_status() == 0
    ah, bh, ch = (t.cpu().numpy() for t in (a, b, want))
    i = batch - 1                                 # one of the cut tiles
    truth = oracle.gemm_f64(N, N, m, n, k, 1.0, ah[i * m * k:], m, bh[i * k * n:], k, 0.0, None, m)
    assert oracle.residual(truth, ch[i * m * n:], m) < oracle.error_threshold(True, k)


@pytest.mark.parametrize("mode,shape,fits", [(FP16TCEC, (256, 256, 8192), True),    # K slices, on the fly
                                             (TF32TCEC, (700, 520, 900), False)])   # panels
def test_nothing_is_allocated_during_a_capture(oracle, monkeypatch, mode, shape, fits):
    """A handle without a workspace, captured.  K slices of the on-the-fly kernel are left out (the
    call needs no memory then); a call that cannot do without panels is refused.  Neither may
    allocate or free, which would end the capture."""
    import torch

    m, n, k = shape
    a, b = oracle.gen_uniform(1, m * k), oracle.gen_uniform(2, k * n)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    c, d = torch.zeros(m * n, device="cuda"), torch.zeros(4, device="cuda")
    monkeypatch.setenv("CUMPSGEMM_STREAM", "0")
    with api.Handle() as h:                       # loads the kernels
        h.use_current_torch_stream()
        h.gemm(N, N, m, n, k, 1.0, da, m, db, k, 0.0, c, m, mode)
        torch.cuda.synchronize()
    with api.Handle() as h:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            h.use_current_torch_stream()
            st = h.gemm(N, N, m, n, k, 1.0, da, m, db, k, 0.0, c, m, mode, check=False)
            d.add_(1.0)                           # the capture goes on
        assert st == (api.CUBLAS_STATUS_SUCCESS if fits else 3)
        c.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert d[0].item() == 1.0
        if fits:
            truth = oracle.gemm_f64(N, N, m, n, k, 1.0, a, m, b, k, 0.0, None, m)
            assert oracle.residual(truth, c.cpu().numpy(), m) < oracle.error_threshold(True, k)
        else:
            assert torch.count_nonzero(c).item() == 0
        del graph
        assert h.kernel_status() == 0


def test_the_limit_decides_about_pieces_and_not_the_history(oracle):
    """K pieces that would go beyond the workspace limit are left out, and the tiles stay whole: with
    the same bits whether or not an earlier call has left a large workspace on the handle."""
    import torch

    batch, m, n, k = 13, 520, 300, 1500           # 78 tiles on 74 pairs: the last four are cut
    a, b = oracle.gen_uniform(1, batch * m * k), oracle.gen_uniform(2, batch * k * n)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()

    def call(h, limit):
        h.set_workspace_limit(limit)
        c = torch.zeros(batch * m * n, device="cuda")
        h.gemm_strided_batch(T, N, m, n, k, 1.0, da, k, m * k, db, k, k * n, 0.0, c, m, m * n, batch,
                             TF32TCEC)
        return c

    with api.Handle() as h:
        h.use_current_torch_stream()
        fresh = call(h, 1 << 20)
        cut = call(h, 0)
        after = call(h, 1 << 20)
        assert torch.equal(fresh, after)
        assert not torch.equal(fresh, cut)
        for c in (fresh, cut):
            res = c.cpu().numpy()
            for i in (0, batch - 1):
                truth = oracle.gemm_f64(T, N, m, n, k, 1.0, a[i * m * k:], k, b[i * k * n:], k, 0.0, None, m)
                assert oracle.residual(truth, res[i * m * n:(i + 1) * m * n], m) < oracle.error_threshold(True, k)
        assert h.kernel_status() == 0


def test_pair_scratch_is_taken_when_needed_and_within_the_limit(oracle, monkeypatch):
    """The pair kernel's scratch for K pieces: none for a launch that cuts no tile (148 tiles are two
    whole waves), none where it would go beyond a workspace limit that the panels keep."""
    import torch

    def used(h, m, n, k, limit, out):
        x = torch.ones(1, device="cuda")          # (the caching allocator's first block)
        a, b = (torch.rand(s, device="cuda", generator=torch.Generator("cuda").manual_seed(9)) * 2 - 1
                for s in (m * k, k * n))
        c = torch.zeros(m * n, device="cuda")
        h.use_current_torch_stream()
        h.set_workspace_limit(limit)
        before = _free_bytes()
        h.gemm(N, N, m, n, k, 1.0, a, m, b, k, 0.0, c, m, FP16TCEC)
        taken = before - _free_bytes()
        out.append(c)
        del x
        return taken

    whole, cut = (9472, 1024, 512), (4096, 4096, 2048)
    panels = lambda m, n, k: 4 * (m + n) * k      # noqa: E731
    outs = []
    for shape in (whole, cut):                    # loads the kernels
        with api.Handle() as h:
            used(h, *shape, 0, outs)
    del outs[:]
    with api.Handle() as h:
        assert used(h, *whole, 0, outs) <= panels(*whole) + SLACK
    with api.Handle() as h:
        assert used(h, *cut, 0, outs) > panels(*cut) + 4 * SLACK
    limit = panels(*cut) + 2 * SLACK
    with api.Handle() as h:
        assert used(h, *cut, limit, outs) <= limit
        assert h.kernel_status() == 0
    monkeypatch.setenv("CUMPSGEMM_TAIL_SPLIT", "0")
    with api.Handle() as h:
        used(h, *cut, 0, outs)
    _, with_pieces, limited, uncut = outs
    assert torch.equal(limited, uncut) and not torch.equal(limited, with_pieces)
