"""Workloads by which the speed of the library is judged.

A case is one call (or the short sequence of calls a program makes) through the public host
interface ``cumpsgemm_b200.api``: column-major FP32 / complex64 operands in device memory, one
handle per process, the stream of the caller.  The sizes are those of the reference's test
(m = n = k = 1024), of ``bench.py`` and of the tests, and generic odd ones; ``draw`` spreads
over the same kinds of call and the whole range between the smallest and the largest.

Fields of a case
  api      "gemm"     one GEMM: ``Handle.gemm``, or ``Handle.gemm_strided_batch`` for batch > 1
           "auto"     statistics of both operands, then the GEMM whose precision the device picks
                      from them (``exp_stats_ext`` twice, ``gemm_strided_batch_with_stats``)
           "explicit" the same decision, with the operands scaled and restored in place by the
                      caller (``scale_A/B/C``, ``reset_scale_A/B``), as code written against the
                      reference's C++ interface does
  complex, op_a, op_b, m, n, k, batch, beta, mode as in the call; pad = elements by which every
  leading dimension exceeds its minimum; dist = how the operands are distributed:
           "uniform"  uniform(-1, 1)
           "scaled"   uniform(-1, 1) * 2^e, e in [-8, 8]
           "wide"     random sign, mantissa in [1, 2), exponent in [-30, 10]
           "tiny"     uniform(-1, 1) * 2^-22
           "normal"   N(0, 1)
           "unit"     Gaussian, every matrix divided by its Frobenius norm (amplitudes of a
                      quantum-circuit state)
"""
import torch

from cumpsgemm_b200 import api

_OPS = {"N": api.CUBLAS_OP_N, "T": api.CUBLAS_OP_T, "C": api.CUBLAS_OP_C}
_LARGEST = 16384  # the headline size, m = n = k

_handle = None


def _get_handle():
    """The one handle a program creates and keeps."""
    global _handle
    if _handle is None:
        _handle = api.Handle()
        _handle.use_current_torch_stream()
    return _handle


def _case(api="gemm", mode="FP16TCEC", m=0, n=0, k=0, op_a="N", op_b="N", batch=1, complex=False,
          beta=0.0, pad=0, dist="uniform", name=None):
    c = dict(api=api, mode=mode, m=m, n=n, k=k, op_a=op_a, op_b=op_b, batch=batch,
             complex=complex, beta=beta, pad=pad, dist=dist)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one small product, called in a loop: launches and host work are most of it
        _case(name="sgemm_128", m=128, n=128, k=128),
        # the reference's own test case and smallest benchmark size
        _case(name="sgemm_1024", m=1024, n=1024, k=1024),
        # ordinary sizes of the benchmark's square sweep, accumulating into C
        _case(name="sgemm_2048", m=2048, n=2048, k=2048, beta=0.5, dist="scaled"),
        _case(name="sgemm_4096_tf32", mode="TF32TCEC", m=4096, n=4096, k=4096, beta=0.5,
              dist="scaled"),
        # nothing a multiple of anything, leading dimensions that rule out vector loads
        _case(name="sgemm_ragged_tn", m=1999, n=3001, k=2777, op_a="T", beta=0.5, pad=1),
        # the headline: the largest square product of the sweep
        _case(name="sgemm_16384", m=_LARGEST, n=_LARGEST, k=_LARGEST, beta=0.5, dist="scaled"),
        # wide exponent range, precision picked on the device (it picks TF32TCEC)
        _case(name="sgemm_8192_auto", api="auto", mode="AUTO", m=8192, n=8192, k=8192,
              dist="wide"),
        # a caller that scales small-magnitude operands itself, weight-gradient shape (op N/T)
        _case(name="sgemm_explicit_nt", api="explicit", mode="AUTO", m=4096, n=1024, k=2048,
              op_b="T", dist="tiny"),
        # quantum-circuit contraction: many small complex products with operand scaling
        _case(name="cgemm_batch_256", mode="FP16TCEC_SCALING", m=256, n=256, k=256, batch=512,
              complex=True, dist="unit"),
        # many small real products
        _case(name="sgemm_batch_128", m=128, n=128, k=128, batch=2048),
        # one complex product with a conjugated operand and complex-accumulate
        _case(name="cgemm_cn", m=1280, n=960, k=1500, op_a="C", complex=True, beta=0.5),
        # inner products of long vectors: few outputs, very long sum
        _case(name="sgemm_long_k", m=256, n=256, k=65536),
    ]


def _log_size(rng, lo, hi):
    """Spread over the logarithm; half of them left as they come, half rounded to a multiple of 32."""
    v = int(round(lo * (hi / lo) ** rng.random()))
    return v if rng.random() < 0.5 else max(lo, (v + 16) // 32 * 32)


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "scaling", "auto", "explicit", "batch", "batch",
                       "long_k"])
    cplx = rng.random() < 0.3
    ops = ["N", "T", "C"] if cplx else ["N", "T"]
    op_a, op_b = rng.choice(ops), rng.choice(ops)
    beta = rng.choice([0.0, 0.5])
    pad = rng.choice([0, 0, 0, 4, 1])
    # (operands of very small magnitude would vanish beside an accumulated C of order one, so they
    # come with beta = 0)
    if kind == "batch":
        m, n, k = (_log_size(rng, 32, 1024) for _ in range(3))
        batch = _log_size(rng, 8, 2048)
        while batch > 8 and batch * max(m * n, m * k, k * n) > 1 << 28:
            batch //= 2
        dist = rng.choice(["uniform", "normal", "unit"])
        return _case(mode=rng.choice(["FP16TCEC", "FP16TCEC", "FP16TCEC_SCALING", "TF32TCEC"]),
                     m=m, n=n, k=k, op_a=op_a, op_b=op_b, batch=batch, complex=cplx,
                     beta=0.0 if dist == "unit" else beta, pad=pad, dist=dist)
    if kind == "long_k":
        return _case(mode=rng.choice(["FP16TCEC", "TF32TCEC"]), m=_log_size(rng, 32, 512),
                     n=_log_size(rng, 32, 512), k=_log_size(rng, 4096, 131072), op_a=op_a,
                     op_b=op_b, complex=cplx, beta=beta, pad=pad)
    m, n, k = (_log_size(rng, 64, 8192) for _ in range(3))
    if kind == "gemm":
        return _case(mode=rng.choice(["FP16TCEC", "FP16TCEC", "TF32TCEC"]), m=m, n=n, k=k,
                     op_a=op_a, op_b=op_b, complex=cplx, beta=beta, pad=pad,
                     dist=rng.choice(["uniform", "scaled", "normal"]))
    if kind == "scaling":
        dist = rng.choice(["tiny", "normal"])
        return _case(mode="FP16TCEC_SCALING", m=m, n=n, k=k, op_a=op_a, op_b=op_b, complex=cplx,
                     beta=0.0 if dist == "tiny" else beta, pad=pad, dist=dist)
    # the explicit sequence un-scales all of C, so it is used with beta = 0
    dist = rng.choice(["tiny", "normal", "scaled"] + (["wide"] if kind == "auto" else []))
    return _case(api=kind, mode="AUTO", m=m, n=n, k=k, op_a=op_a, op_b=op_b, complex=cplx,
                 beta=0.0 if kind == "explicit" or dist == "tiny" else beta, pad=pad, dist=dist)


def _values(shape, dist, cplx, gen):
    dev = torch.device("cuda")

    def uniform(s):
        return torch.rand(s, device=dev, generator=gen).mul_(2).sub_(1)

    def exponent(s, lo, hi):
        return torch.randint(lo, hi + 1, s, device=dev, generator=gen, dtype=torch.int32)

    real = tuple(shape) + ((2,) if cplx else ())
    if dist == "scaled":
        x = torch.ldexp(uniform(real), exponent(real, -8, 8))
    elif dist == "wide":
        x = torch.ldexp(torch.rand(real, device=dev, generator=gen).add_(1), exponent(real, -30, 10))
        x = torch.where(uniform(real) < 0, -x, x)
    elif dist == "tiny":
        x = uniform(real).mul_(2.0 ** -22)
    elif dist in ("normal", "unit"):
        x = torch.randn(real, device=dev, generator=gen)
        if dist == "unit":
            x /= x.flatten(1).norm(dim=1).reshape((-1,) + (1,) * (x.dim() - 1))
    else:
        x = uniform(real)
    return torch.view_as_complex(x) if cplx else x


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    c = case
    rows_a, cols_a = (c["m"], c["k"]) if c["op_a"] == "N" else (c["k"], c["m"])
    rows_b, cols_b = (c["k"], c["n"]) if c["op_b"] == "N" else (c["n"], c["k"])
    lda, ldb, ldc = rows_a + c["pad"], rows_b + c["pad"], c["m"] + c["pad"]
    # column-major: the leading dimension is the last one of the tensor
    A = _values((c["batch"], cols_a, lda), c["dist"], c["complex"], gen)
    B = _values((c["batch"], cols_b, ldb), c["dist"], c["complex"], gen)
    if c["beta"] != 0:
        C = _values((c["batch"], c["n"], ldc), "uniform", c["complex"], gen)
    else:
        C = torch.zeros((c["batch"], c["n"], ldc), device="cuda",
                        dtype=torch.complex64 if c["complex"] else torch.float32)
    alpha = 1.0
    if c["complex"]:
        alpha = 0.75 - 0.5j
    return dict(h=_get_handle(), case=c, A=A, B=B, C=C, rows_a=rows_a, cols_a=cols_a,
                rows_b=rows_b, cols_b=cols_b, lda=lda, ldb=ldb, ldc=ldc, alpha=alpha,
                op_a=_OPS[c["op_a"]], op_b=_OPS[c["op_b"]], mode=api.ComputeMode[c["mode"]])


def run(state):
    s, c = state, state["case"]
    h, A, B, C = s["h"], s["A"], s["B"], s["C"]
    m, n, k, batch, beta = c["m"], c["n"], c["k"], c["batch"], c["beta"]
    stride_a, stride_b, stride_c = s["lda"] * s["cols_a"], s["ldb"] * s["cols_b"], s["ldc"] * n
    if c["api"] == "gemm":
        if batch == 1:
            h.gemm(s["op_a"], s["op_b"], m, n, k, s["alpha"], A, s["lda"], B, s["ldb"], beta, C,
                   s["ldc"], s["mode"])
        else:
            h.gemm_strided_batch(s["op_a"], s["op_b"], m, n, k, s["alpha"], A, s["lda"], stride_a,
                                 B, s["ldb"], stride_b, beta, C, s["ldc"], stride_c, batch,
                                 s["mode"])
        return C
    id_a = h.exp_stats_ext(s["rows_a"], s["cols_a"], A, s["lda"])
    id_b = h.exp_stats_ext(s["rows_b"], s["cols_b"], B, s["ldb"])
    if c["api"] == "auto":
        h.gemm_strided_batch_with_stats(s["op_a"], s["op_b"], m, n, k, s["alpha"], A, s["lda"], 0,
                                        B, s["ldb"], 0, beta, C, s["ldc"], 0, 1, s["mode"], id_a,
                                        id_b)
        return C
    flag = h.get_next_dynamic_launch_buffer_id()
    h.set_dynamic_launch_buffer_by_exp_stats(flag, id_a, id_b)
    h.scale_A(id_a, flag, s["rows_a"], s["cols_a"], A, s["lda"])
    h.scale_B(id_b, flag, s["rows_b"], s["cols_b"], B, s["ldb"])
    h.set_dynamic_launch_flag_buffer_id(flag)
    h.gemm(s["op_a"], s["op_b"], m, n, k, s["alpha"], A, s["lda"], B, s["ldb"], 0.0, C, s["ldc"],
           s["mode"])
    h.unset_dynamic_launch_flag_buffer_id()
    h.scale_C(id_a, id_b, flag, m, n, C, s["ldc"])
    h.reset_scale_A(id_a, flag, s["rows_a"], s["cols_a"], A, s["lda"])
    h.reset_scale_B(id_b, flag, s["rows_b"], s["cols_b"], B, s["ldb"])
    return [C, A, B]


def work(case):
    """Operands read once, C written once (and read when it is accumulated into); 2 m n k
    floating-point operations per real product, 8 m n k per complex one.  The statistics and the
    in-place scaling need no further pass over memory in principle, so they add nothing here."""
    c = case
    size = 8 if c["complex"] else 4
    words = c["m"] * c["k"] + c["k"] * c["n"] + c["m"] * c["n"] * (2 if c["beta"] != 0 else 1)
    per = (8.0 if c["complex"] else 2.0) * c["m"] * c["n"] * c["k"]
    if c["api"] == "explicit":  # the caller asked for the scaled and restored operands in memory
        words += c["m"] * c["k"] + c["k"] * c["n"]
    return {"bytes": float(c["batch"] * size * words), "flops": float(c["batch"] * per)}


def tolerance(case):
    # Every mode gives FP32-level results.  Against a product formed in 64 bits the listed cases and
    # forty drawn ones show at most 4.1e-7 (2-norm) and 2.6e-6 (largest); four to five times that.
    return {"rel": 2e-6, "max": 1.2e-5}
