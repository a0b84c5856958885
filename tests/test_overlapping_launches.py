"""Kernels that may start under the tail of the kernel that writes their operands (launch_dependent) read them with ordinary loads:
the non-coherent ones (__ldg, ld.global.nc, const __restrict__ parameters) want memory that is read-only for the kernel's whole life."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mp-sparse-attn_b200", "csrc")
NON_COHERENT = re.compile(r"__ldg\b|ld\.global(\.\w+)*\.nc\b|__restrict__")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"/\*.*?\*/|//[^\n]*", "", text, flags=re.S)


def _first_launches(code):
    """Names of the kernels whose launch overlaps whatever is before it on the stream."""
    flags = set(re.findall(r"bool (\w+) = [^;]*overlaps_previous\(", code)) | {r"overlaps_previous\(st\)"}
    names = set()
    for call in re.findall(r"launch_dependent\((.*?)\);", code, flags=re.S):
        if any(re.search(r"\b" + f, call) for f in flags):
            names.add(re.match(r"\s*(\w+)", call).group(1))
    return names


def test_operands_of_overlapping_launches_are_read_coherently():
    found = set()
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        code = _code(name)
        first = _first_launches(code)
        found |= first
        if not first:
            continue
        if name == "quant.cu":                            # other kernels of this file start after their predecessor's end
            assert first == {"col_sum_kernel"}
            body = re.search(r"\bcol_sum_kernel\(const T\* x.*?\n}\n", code, flags=re.S).group(0)
        else:
            body = code
        assert "grid_dependency_wait()" in body
        assert not NON_COHERENT.search(body), name
    assert found == {"col_sum_kernel", "prep_kernel", "kernel"}, found      # ("kernel": the product's local name for its instance)
