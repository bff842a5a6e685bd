"""Gradients of training attention, whose two last kernels run beside one another (csrc/attention_bwd_tc.cu): the next kernels on the stream see both."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,heads,kv", [([1], 12, 2), ([700, 130], 12, 2), ([64] * 9, 28, 4), ([3000], 12, 2), ([1500, 40, 900], 28, 4)])
def test_readers_behind_the_backward_see_all_gradients(lens, heads, kv):
    from nanorlhf_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(0)
    T = sum(lens)
    q, k, v, do = (torch.randn(T, h, 128, generator=g, device="cuda").bfloat16() for h in (heads, kv, kv, heads))
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    w = torch.randn(kv * 128, kv * 128, generator=g, device="cuda").bfloat16()

    def run():
        from nanorlhf_b200.ops import gemm
        o = ops.attention_varlen(*leaves, cu, max(lens))
        dq, dk, dv = torch.autograd.grad(o, leaves, do)
        # readers at once, one of them launched over the end of the backward, and buffers that take the place of freed ones
        return gemm.gemm(dk.view(T, -1), w), dv.clone(), dq.clone(), dk

    first = run()
    torch.cuda.synchronize()
    assert all(torch.isfinite(t).all() for t in first)
    for _ in range(20):
        again = run()
        assert all(torch.equal(a, b) for a, b in zip(first, again))
