"""A kernel that is launched to begin under the end of the one before it must wait for it before it touches memory.  Read
off the sources, since what comes too early seldom shows."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megalodon_b200", "csrc")


def _sources():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            yield f, re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())


def _bodies(text):
    """{kernel: what follows its opening brace}"""
    found = {}
    for m in re.finditer(r"__global__", text):
        depth, name, i = 0, None, m.end()
        while text[i] not in "{;" or depth:
            if text[i] == "(" and depth == 0:
                name = re.search(r"(\w+)\s*$", text[m.end():i]).group(1)
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        if text[i] == "{":
            found[name] = text[i + 1:]
    return found


def _launched():
    out = []
    for f, text in _sources():
        bodies = _bodies(text)
        for name in sorted(set(re.findall(r"launch_dependent\(\s*(\w+)", text))):
            if name in bodies:
                out.append((f, name, bodies[name], True))
                continue
            # a variable: the kernels that it is set to anywhere in the file (the products, which prepare before they wait)
            kernels = sorted(set(re.findall(rf"\b{name}\s*=\s*(\w+)", text)))
            assert kernels and all(k in bodies for k in kernels), (f, name, kernels)
            out += [(f, k, bodies[k], False) for k in kernels]
    return out


def test_the_launches_are_found():
    found = {(f, name) for f, name, _, _ in _launched()}
    assert len(found) >= 40
    assert {("gemm_sm100.cu", "gemm_tcgen05_kernel"), ("gemm_sm100.cu", "gemm_tcgen05_pair_kernel")} <= found
    # (the launcher's own text is not among the sources) every launch names a kernel or a variable of its file
    assert all(re.match(r"[A-Za-z_]\w*\s*[<,]", m) for _, t in _sources() for m in re.findall(r"launch_dependent\(\s*([^;]{1,60})", t))


@pytest.mark.parametrize("file,name,body,first", _launched(), ids=lambda v: v if isinstance(v, str) and len(v) < 45 else "")
def test_kernels_wait_before_they_touch_memory(file, name, body, first):
    if first:
        assert body.lstrip().startswith("begin_dependent();")
    else:
        before = body[:body.index("begin_dependent();")]
        assert not re.search(r"tma_load|p\.C\b|__ldc|epi_staged|epi_direct|p\.bias|gather_copy_warp\(", before)
