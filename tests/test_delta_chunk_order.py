"""The chunked delta-rule scan zeroes its staging memory with ordinary stores before bulk copies write there.  Nothing but a proxy fence of the
storing threads orders the two, and which comes first in a run is not ours to choose: read from the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanorlhf_b200", "csrc")


def test_zeros_are_fenced_before_the_copies():
    with open(os.path.join(CSRC, "delta_chunk_tc.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    zeros, copies = re.search(r"all\[x\]\s*=\s*0\.f;", src).end(), src.rindex("bulk_load(raw")
    between = src[zeros:copies]
    # statements of all the storing threads, in this order: fence, then the barrier behind which one warp issues the copies
    assert re.match(r"\s*fence_proxy_async_smem\(\);\s*named_barrier_sync\(1, kDcLoaders\);", between)


def test_a_blocks_place_on_the_line_is_the_order_of_its_start():
    """A block waits for its neighbour's state.  CUDA does not say in which order blocks start, so the place comes from a counter that each takes when it runs."""
    with open(os.path.join(CSRC, "delta_chunk_tc.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    assert re.search(r"\*ticket = atomicAdd\(p\.line\.ticket, 1\);", src) and re.search(r"auto line = \[&\]\(\) \{[^}]*\*ticket; \};", src)
    assert not re.search(r"blockIdx[^;]*line|line[^;]*blockIdx", src) and src.count("*l.ticket = 0;") == 1
