"""When the head's forward leaves its logits for the backward: never where that would take memory that others hold or a step may need."""
import pytest

from nanorlhf_b200 import _C

G = 1 << 30


@pytest.mark.parametrize("M,V", [(100, 151936), (6001, 151936), (7067, 151936), (65536, 16384), (1, 8)])
@pytest.mark.parametrize("total", [180 * G, 80 * G])
def test_a_quarter_of_the_device_stays(M, V, total):
    line = total // 4 * 3 - 8 * M * V
    assert _C.lmhead_keeps_logits(M, V, 0, total) and _C.lmhead_keeps_logits(M, V, line, total)
    assert not _C.lmhead_keeps_logits(M, V, line + 1, total) and not _C.lmhead_keeps_logits(M, V, total, total)


@pytest.mark.parametrize("M,V", [(0, 1024), (7068, 151936), (65536, 16392), (5, 1004), (1 << 40, 1 << 20)])
def test_sizes_that_keep_nothing(M, V):
    assert not _C.lmhead_keeps_logits(M, V, 0, 180 * G)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [64, 600])
def test_memory_that_is_only_reserved_counts(rows):
    import torch
    V = 151936
    h = torch.empty(rows, 8, dtype=torch.bfloat16, device="cuda")
    torch.cuda.empty_cache()
    assert _C.lmhead_logits_buffer(h, V) is not None
    x = torch.empty(torch.cuda.mem_get_info()[1] // 4 * 3, dtype=torch.uint8, device="cuda")
    del x                                                        # stays with the allocator
    assert torch.cuda.memory_allocated() < G and _C.lmhead_logits_buffer(h, V) is None
    torch.cuda.empty_cache()
    assert _C.lmhead_logits_buffer(h, V).shape == (rows, V)


@pytest.mark.gpu
def test_a_captured_step_asks_too():
    import torch

    from nanorlhf_b200 import ops
    h = torch.randn(600, 64, device="cuda").bfloat16().requires_grad_()
    w, t = torch.randn(151936, 64, device="cuda").bfloat16(), torch.zeros(600, dtype=torch.long, device="cuda")

    def step():
        lp, _ = ops.lmhead_logprob(h, w, t, 1.0, False)
        return torch.autograd.grad(lp.sum(), h)[0]
    want = step()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        got = step()
    graph.replay()
    assert torch.equal(got, want)


@pytest.mark.gpu
def test_the_driver_is_not_asked_while_nothing_is_reserved():
    """It may take milliseconds to answer."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    from nanorlhf_b200 import ops
    h = torch.randn(600, 64, device="cuda").bfloat16().requires_grad_()
    w, t = torch.randn(151936, 64, device="cuda").bfloat16(), torch.zeros(600, dtype=torch.long, device="cuda")

    def step():
        lp, _ = ops.lmhead_logprob(h, w, t, 1.0, False)
        return torch.autograd.grad(lp.sum(), h)[0]

    def asked(f):
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            f()
            torch.cuda.synchronize()
        return sum(e.name == "cudaMemGetInfo" for e in p.events())
    step()
    step()
    if asked(torch.cuda.mem_get_info) == 0:
        pytest.skip("the profiler does not show such calls")
    assert asked(lambda: [step() for _ in range(3)]) == 0
