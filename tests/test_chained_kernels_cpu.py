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
