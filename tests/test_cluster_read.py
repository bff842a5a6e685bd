"""Shared memory of a cluster's other blocks is read behind a barrier at which all have arrived with their data, and in front of one that all wait at
before they leave: read from the sources, as the order of the blocks is not ours to choose."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanorlhf_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_the_header_only_reads():
    src = _source("cluster_read.h")
    assert "ld.shared::cluster" in src and not re.search(r"\b(st|st\.async|red|atom|cp)\.[\w.:]*shared::cluster", src)
    assert {f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and "cluster_read.h" in _source(f)} == {"gemm_tc.cu"}


def test_gemm_parts_are_read_between_two_barriers():
    src = _source("gemm_tc.cu")
    section = src[src.index("  if (CLUSTER) {", src.index("tma_store_wait<0>();\n  }")):]
    barrier, first, last = section.index("cluster_sync_all();"), section.index("ld_cluster_f4("), section.rindex("ld_cluster_f4(")
    assert 0 < barrier < first
    after = section[last:]
    assert "if (CLUSTER) cluster_sync_all();" in after and after.index("if (CLUSTER) cluster_sync_all();") < after.index("tmem_dealloc_cg")
    assert "return" not in section[:section.index("tmem_dealloc_cg")]
