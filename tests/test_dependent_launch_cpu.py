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
            if name == "kern":                             # (the products, whose kernels prepare before they wait)
                out += [(f, k, b, False) for k, b in bodies.items() if k.startswith("gemm_tcgen05")]
            else:
                out.append((f, name, bodies[name], True))
    return out


def test_the_launches_are_found():
    assert len(_launched()) > 40


@pytest.mark.parametrize("file,name,body,first", _launched(), ids=lambda v: v if isinstance(v, str) and len(v) < 45 else "")
def test_kernels_wait_before_they_touch_memory(file, name, body, first):
    if first:
        assert body.lstrip().startswith("begin_dependent();")
    else:
        before = body[:body.index("begin_dependent();")]
        assert not re.search(r"tma_load|p\.C\b|__ldc|epi_staged|epi_direct|p\.bias|gather_copy_warp\(", before)
