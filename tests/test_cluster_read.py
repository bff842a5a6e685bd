"""Shared memory of a cluster's other blocks is read behind a barrier at which all have arrived with their data, and in front of one that all wait at
before they leave: read from the sources, as the order of the blocks is not ours to choose."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanorlhf_b200", "csrc")


def _source(name):
    """A file without comments, blanks and line ends."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"\s+", "", re.sub(r"//[^\n]*", "", f.read()))


def _body(src, name):
    """Body of the function that is defined as ``name``."""
    at = re.search(r"(?<!\w)\w*" + name + r"\([^;{]*\)\{", src).end()
    depth, i = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        i += 1
    return src[at:i - 1]


def test_the_header_only_reads():
    src = _source("cluster_read.h")
    assert "ld.shared::cluster" in src and not re.search(r"(st|red|atom|cp)\.[\w.:]*shared::cluster", src)
    assert {f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h", ".cpp")) and "cluster_read.h" in _source(f)} == {"gemm_tc.cu"}


def test_gemm_parts_are_read_between_two_barriers():
    src = _source("gemm_tc.cu")
    body = _body(src, "gemm_tc_body")
    first, last = body.index("ld_cluster_f4("), body.rindex("ld_cluster_f4(")
    assert src.count("ld_cluster_f4(") == body.count("ld_cluster_f4(")               # nowhere else
    written = body.index("if(CLUSTER){")                                             # where a block leaves its part
    branch = body.index("if(CLUSTER){", written + 1)                                 # all threads of it come here
    assert written < branch < body.index("cluster_sync_all();", branch) < first
    assert not re.search(r"[{};](if|for|while)\(", body[branch + len("if(CLUSTER){") - 1:body.index("cluster_sync_all();", branch)])
    leave = body.index("if(CLUSTER)cluster_sync_all();", last)
    assert last < leave < body.index("tmem_dealloc_cg", last)
    assert "return;" not in body[branch:leave]
