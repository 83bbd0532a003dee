"""Distributed shared memory may be touched only once the CTA that owns it has started, which a cluster barrier shows.
Read off the kernels' source, since a CTA that is late is nothing a test can bring about."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megalodon_b200", "csrc")


def _kernels():
    """(file, name, body) of every kernel that addresses another CTA's shared memory."""
    found = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__", text):
            depth, name, i = 0, None, m.end()
            while text[i] not in "{;":                   # the signature: the last word before a bracket at its top level
                if text[i] == "(" and depth == 0:
                    name = re.search(r"(\w+)\s*$", text[m.end():i]).group(1)
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            start, depth = i, 0
            while text[i] != ";" or depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            if "map_to_cta(" in text[start:i]:
                found.append((f, name, text[start:i]))
    return found


def test_the_kernels_are_found():
    assert {"decode_norm_ema_kernel", "skinny_gemm_kernel", "gemm_tcgen05_pair_kernel"} <= {n for _, n, _ in _kernels()}


@pytest.mark.parametrize("file,name,body", _kernels(), ids=lambda v: v if isinstance(v, str) and len(v) < 40 else "")
def test_a_cluster_barrier_precedes_the_first_remote_access(file, name, body):
    before = [""]                                        # what precedes the access in the blocks that enclose it
    for c in body[:body.index("map_to_cta(")]:
        if c == "{":
            before.append("")
        elif c == "}":
            before.pop()
        else:
            before[-1] += c
    before = " ".join(before)
    assert "cluster_wait()" in before or "cluster_sync_all()" in before, f"{file}: {name}"
