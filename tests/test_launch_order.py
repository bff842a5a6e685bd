"""Kernels that start before the kernel in front has ended (csrc/launch.h) wait for it in every thread, and let the next one start only behind that wait.
Whether a kernel that does not would read old values is not ours to choose, so this is read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanorlhf_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _body(src, name):
    """Body of the function that is defined as ``name``."""
    at = re.search(r"\b" + name + r"\s*\([^;{]*\)\s*\{", src).end()
    depth, i = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        i += 1
    return src[at:i - 1]


def _unconditional(body):
    """The statements of a body that are in no block of their own."""
    out, depth = [], 0
    for c in body:
        depth -= c == "}"
        if depth == 0:
            out.append(c)
        depth += c == "{"
    return "".join(out)


def _launched(src):
    """Kernels that a file launches this way, by name or through a variable."""
    names = set()
    for a in re.findall(r"launch_(?:dependent(?:_clusters)?\(|early_if\(early,)\s*(\w+)", src):
        names |= set(re.findall(r"\b" + a + r"\s*=\s*(\w+_kernel)\b", src)) or {a}
    return names


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "launch_dependent" in _source(f))


def test_the_files_are_found():
    assert {"gemm_tc.cu", "elementwise.cu", "attention_fwd_tc.cu", "attention_bwd_tc.cu", "attention_decode.cu"} <= set(FILES)


@pytest.mark.parametrize("name", FILES)
def test_kernels_wait_before_they_let_the_next_one_start(name):
    src = _source(name)
    kernels = _launched(src)
    assert kernels
    for k in kernels:
        body = _body(src, k)
        if "gemm_tc_body<" in body:                                       # all that such a kernel does
            body = _body(src, "gemm_tc_body")
        flat = _unconditional(body)
        wait = re.search(r"(^|[;{}])\s*pdl_wait\(\);", flat)
        assert wait, k
        assert "return" not in flat[:wait.start()] and "pdl_launch_dependents" not in body[:body.index("pdl_wait();")], k
