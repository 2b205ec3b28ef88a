"""Source rule of the programmatic launches (no GPU needed): a kernel that may be resident while its predecessor in the
stream still writes reads that predecessor's data with coherent loads.  The read-only path (`__ldg`, or a `const
__restrict__` pointer the compiler may turn into it) is for data that is constant while the kernel lives."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "skyrl-tx-rocm_b200" / "csrc"


def _kernel(source, name):
    text = (CSRC / source).read_text()
    at = re.search(rf"\b{name}\(", text)
    head_end = text.index("{", at.end())
    depth, i = 1, head_end + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[at.end():head_end], text[head_end:i]


@pytest.mark.parametrize("source,name,written_before,constant", [
    ("quant_route_sm100.cu", "rms_quant_kernel", ("x", "row_map"), ()),
    ("quant_route_sm100.cu", "quant_stream_kernel", ("x", "row_amax"), ()),
    ("grad_quant_sm100.cu", "grad_quant_kernel", ("dy", "row_map"), ("cs",)),
    ("grouped_gemm_sm100.cu", "group_quant_kernel", ("x", "row_map"), ()),
])
def test_quantisers_read_their_input_coherently(source, name, written_before, constant):
    params, body = _kernel(source, name)
    for p in written_before:
        decl = re.search(rf"const [\w ]+\*\s*(__restrict__\s+)?{p}\b", params)
        assert decl and decl.group(1) is None, f"{name}: {p} must not be const __restrict__"
        assert not re.search(rf"\b{p}\[", body), f"{name}: {p} is indexed directly"
    for arg in re.findall(r"__ldg\(\s*(\w+)", body):
        assert arg in constant, f"{name}: __ldg({arg} ...)"


def test_gemms_read_the_activation_scales_coherently():
    for source in ("w8a8_gemm_sm100.cu", "grouped_gemm_sm100.cu", "planes_gemm_sm100.cu"):
        assert not re.search(r"__ldg\(\s*(p\.sx|p\.s|sxp)\b", (CSRC / source).read_text()), source
