"""Kernels that are launched behind the previous kernel of the stream (programmatic serialization)
may start before it ends: whatever an earlier kernel writes is read behind griddepcontrol.wait.
Checked on the source text of the GEMM kernels, for the record an AUTO / FP16TCEC_SCALING call
decides on the device (a wrong order shows on a GPU only by chance)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cumpsgemm_b200" / "csrc"


def _body(text, name):
    """The body of the function definition called `name`, comments removed."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(rf"\b{name}\(", text):
        i, depth = m.end(), 1
        while depth:                              # past the parameter list
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        if not text[i:].lstrip().startswith("{"):
            continue                              # a call or a declaration
        i = start = text.index("{", i) + 1
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        return text[start:i]
    raise AssertionError(f"{name} is not defined")


@pytest.mark.parametrize("source,functions", [
    ("tcec_gemm.cu", ["tcec_gemm_body", "tcec_gemm_auto_kernel"]),
    ("tcec_gemm_pair.cu", ["pair_body", "tcec_gemm_pair_auto_kernel"]),
    ("tcec_gemm_stream.cu", ["stream_body", "tcec_gemm_stream_kernel"])])
def test_device_decision_is_read_behind_the_wait(source, functions):
    text = (CSRC / source).read_text()
    for name in functions:
        body = _body(text, name)
        assert "dyn->" in body, name
        assert "griddep_wait()" in body, name
        assert body.index("griddep_wait()") < body.index("dyn->"), name


@pytest.mark.parametrize("source,function,wait", [
    ("tcec_gemm_stream.cu", "tcec_gemm_stream_solo_kernel", "griddep_wait()"),
    ("tcec_gemm_small.cu", "tcec_gemm_small_kernel", "CUMPSGEMM_CHAINED_KERNEL_ENTRY()")])
def test_device_decision_is_read_behind_the_wait_on_single_ctas(source, function, wait):
    body = _body((CSRC / source).read_text(), function)
    assert body.index(wait) < body.index("dyn->")
    if function == "tcec_gemm_small_kernel":      # all that touches global memory is behind it
        assert body.index(wait) < body.index("small_body<")


@pytest.mark.parametrize("source", ["tcec_gemm.cu", "tcec_gemm_pair.cu", "tcec_gemm_fused.cu",
                                    "tcec_gemm_small.cu", "tcec_gemm_stream.cu"])
def test_a_warp_that_waits_for_an_accumulator_goes_on_as_a_whole(source):
    """A bounded wait gives up lane by lane; the loads from tensor memory that follow need the whole
    warp, so its lanes agree on the result (likewise converters that write to tensor memory)."""
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    waits = [s for s in re.findall(r"[^;{}]*ptx::mbar_wait[^;]*;", text)
             if "kErrWaitD0Full" in s or "kErrWaitD1Full" in s]
    assert waits
    if source == "tcec_gemm_stream.cu":
        waits += re.findall(r"[^;{}]*ptx::mbar_wait[^;{}]*;", _body(text, "convert_loop"))[:1]
    for s in waits:
        assert "warp_agrees(" in s, s


def test_the_on_the_fly_kernel_chooses_its_stores_warp_by_warp():
    """Its general epilogue exchanges values between the lanes of a warp: no lane may take the short one
    by itself (a warp that holds the last rows of a matrix would wait for it without a limit)."""
    body = _body((CSRC / "tcec_gemm_fused.cu").read_text(), "tcec_gemm_fused_kernel")
    short = re.search(r"if \(plain\b([^{]*)\{", body).group(1)
    assert "__shfl_xor_sync(0xffffffffu" in body and "__all_sync(0xffffffffu, row_ok)" in short
    assert "row_ok" not in short.replace("__all_sync(0xffffffffu, row_ok)", "")
