"""A block's shared memory may be written by its cluster's other blocks only once it is known to have started.  The order of start-up is not
ours to choose, so this is read from the sources: every remote write follows a cluster barrier that all blocks arrive at on entry.  Remote reads have a
header of their own (test_cluster_read.py)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanorlhf_b200", "csrc")
REMOTE = re.compile(r"map_shared_rank\(|mapa\.shared::cluster")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _function(src, name):
    """Body of the function that is defined as ``name``."""
    at = re.search(r"\b" + name + r"\s*\([^;{]*\)\s*\{", src).end()
    depth, i = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        i += 1
    return src[at:i]


def test_no_other_file_writes_remote_shared_memory():
    reach = {f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h", ".cpp")) and REMOTE.search(_source(f))}
    assert reach == {"rl_kernels.cu", "sampling.cu", "cluster_read.h"}


@pytest.mark.parametrize("kernel", ["policy_loss_kernel", "value_loss_kernel"])
def test_losses_wait_for_the_start_of_the_cluster(kernel):
    src = _source("rl_kernels.cu")
    body, sums = _function(src, kernel), _function(src, "loss_sums")
    assert body.lstrip().startswith("if (scratch == nullptr) cluster_started_arrive();") and "loss_sums(s, scratch, t)" in body
    assert 0 <= sums.find("cluster_started_wait()") < sums.find("map_shared_rank")
    assert "return" not in body[:body.find("loss_sums(")].replace("if (!", "")      # every thread that arrives also waits


def test_sampler_waits_for_the_start_of_the_cluster():
    body = _function(_source("sampling.cu"), "sample_top_p_smem_kernel")
    arrive, wait, first = (body.find(s) for s in ("barrier.cluster.arrive", "barrier.cluster.wait", "cluster_publish("))
    assert 0 <= arrive < wait < first
