"""The split pass on sources whose rows are not 16-byte aligned, and pair tiles whose K ranges are
shared by all CTA pairs, against the FP64 oracle (pass criterion of the other GEMM tests)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from cumpsgemm_b200 import api  # noqa: E402

N, T, Cj = api.CUBLAS_OP_N, api.CUBLAS_OP_T, api.CUBLAS_OP_C
FP16TCEC, TF32TCEC = api.ComputeMode.FP16TCEC, api.ComputeMode.TF32TCEC


def _run(handle, oracle, cplx, op_a, op_b, m, n, k, mode, beta, pad, offset=0, truth=True):
    import torch

    def gen(seed, count):
        x = oracle.gen_uniform(seed, count)
        return (x + 1j * oracle.gen_uniform(seed + 100, count)).astype(np.complex64) if cplx else x

    am, an = (m, k) if op_a == N else (k, m)
    bm, bn = (k, n) if op_b == N else (n, k)
    lda, ldb, ldc = am + pad, bm + pad, m + pad
    a, b, c0 = gen(1, lda * an + offset), gen(2, ldb * bn + offset), gen(3, ldc * n)
    alpha = 0.75 - 0.5j if cplx else 1.25
    da, db, dc = (torch.from_numpy(x.copy()).cuda() for x in (a, b, c0))
    handle.gemm(op_a, op_b, m, n, k, alpha, da[offset:], lda, db[offset:], ldb, beta, dc, ldc, mode)
    res = dc.cpu().numpy()
    if truth:
        want = oracle.gemm_f64(op_a, op_b, m, n, k, alpha, a[offset:], lda, b[offset:], ldb, beta, c0, ldc)
        assert oracle.residual(want, res, ldc) < oracle.error_threshold(True, k * (2 if cplx else 1))
    return res


@pytest.mark.parametrize("mode", [FP16TCEC, TF32TCEC])
@pytest.mark.parametrize("op_a,op_b", [(N, N), (N, T), (T, N), (T, T)])
@pytest.mark.parametrize("size", [(63, 65, 64), (64, 1, 129), (130, 67, 1), (257, 190, 95)])
def test_unaligned_sources(handle, oracle, mode, op_a, op_b, size):
    """Odd leading dimensions, a base address that is only 4-byte aligned, and both aligned."""
    m, n, k = size
    _run(handle, oracle, False, op_a, op_b, m, n, k, mode, 0.5, pad=1, offset=1)
    _run(handle, oracle, False, op_a, op_b, m, n, k, mode, 0.0, pad=3)
    _run(handle, oracle, False, op_a, op_b, 64, 68, 72, mode, 0.5, pad=0)


@pytest.mark.parametrize("cplx,op_a,mode", [(False, T, TF32TCEC), (True, Cj, FP16TCEC)])
def test_pair_tiles_shared_by_all_pairs(handle, oracle, cplx, op_a, mode):
    """40 tiles on 74 pairs: more than half a wave, so the k range of all tiles is cut into 74
    equal pieces, most tiles into two or three, added by a second kernel.  Right, bit-identical
    from run to run, and different from the uncut sum."""
    m, n, k = (1280, 1000, 1600) if cplx else (2560, 1000, 1600)
    os.environ["CUMPSGEMM_PAIR"] = "1"
    try:
        handle.reload_tuning_env()
        outs = [_run(handle, oracle, cplx, op_a, N, m, n, k, mode, -0.5, pad=1, truth=i == 0)
                for i in range(2)]
        np.testing.assert_array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))
        os.environ["CUMPSGEMM_TAIL_SPLIT"] = "0"
        handle.reload_tuning_env()
        uncut = _run(handle, oracle, cplx, op_a, N, m, n, k, mode, -0.5, pad=1)
        assert not np.array_equal(uncut.view(np.uint32), outs[0].view(np.uint32))
    finally:
        os.environ.pop("CUMPSGEMM_PAIR", None)
        os.environ.pop("CUMPSGEMM_TAIL_SPLIT", None)
        handle.reload_tuning_env()


def test_capture_without_room_for_pieces(oracle):
    """A call whose K pieces would need workspace memory, captured into a graph on a handle that has
    none: no allocation may happen, so the tiles stay whole, and the replay is right."""
    import torch

    batch, m, n, k = 13, 520, 300, 1500           # 78 tiles on 74 pairs: the last four would be cut
    a, b = oracle.gen_uniform(1, batch * m * k), oracle.gen_uniform(2, batch * k * n)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    dc = torch.zeros(batch * m * n, device="cuda")
    with api.Handle() as h:
        s = torch.cuda.Stream()
        # one call of another size on this stream first: library set-up is not part of the test
        with torch.cuda.stream(s):
            h.set_stream(s)
            h.gemm_strided_batch(T, N, 256, 256, 64, 1.0, da, 64, 256 * 64, db, 64, 256 * 64, 0.0, dc,
                                 256, 256 * 256, 8, FP16TCEC)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            h.gemm_strided_batch(T, N, m, n, k, 1.0, da, k, m * k, db, k, k * n, 0.0, dc, m, m * n,
                                 batch, FP16TCEC)
            assert h.last_route() == (api.ROUTE_STREAMING, False)
        g.replay()
        torch.cuda.synchronize()
        res = dc.cpu().numpy()
        for i in (0, batch - 1):
            want = oracle.gemm_f64(T, N, m, n, k, 1.0, a[i * m * k:], k, b[i * k * n:], k, 0.0, None, m)
            assert oracle.residual(want, res[i * m * n:(i + 1) * m * n], m) < oracle.error_threshold(True, k)
        with torch.cuda.stream(s):                # (with memory to be had they are)
            h.gemm_strided_batch(T, N, m, n, k, 1.0, da, k, m * k, db, k, k * n, 0.0, dc, m, m * n,
                                 batch, FP16TCEC)
            assert h.last_route() == (api.ROUTE_STREAMING, True)
        assert h.kernel_status() == 0
        del g


def test_the_first_chunk_of_the_pair_kernel_can_be_lengthened(handle, oracle, monkeypatch):
    """CUMPSGEMM_FIRST_CHUNK sets how many stages the pair kernel sums up before it drains its
    accumulator for the first time in a tile: another rounding, the same result within tolerance; a
    value below the drain chunk changes nothing."""
    args = (handle, oracle, False, N, N, 520, 300, 1500, FP16TCEC, 0.5, 0)
    monkeypatch.setenv("CUMPSGEMM_PAIR", "1")
    monkeypatch.setenv("CUMPSGEMM_TAIL_SPLIT", "0")
    monkeypatch.setenv("CUMPSGEMM_DRAIN_CHUNK", "2")
    outs = {}
    for first in ("0", "1", "7", "1000"):         # default, below the drain chunk, odd, whole K loop
        monkeypatch.setenv("CUMPSGEMM_FIRST_CHUNK", first)
        handle.reload_tuning_env()
        outs[first] = _run(*args).view(np.uint32)
    for name in ("PAIR", "TAIL_SPLIT", "DRAIN_CHUNK", "FIRST_CHUNK"):
        monkeypatch.delenv("CUMPSGEMM_" + name)
    handle.reload_tuning_env()
    np.testing.assert_array_equal(outs["0"], outs["1"])
    assert not np.array_equal(outs["0"], outs["7"])
    assert not np.array_equal(outs["7"], outs["1000"])
