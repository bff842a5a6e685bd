"""A traced program that holds a loss follows its inputs, and the loss's gradient with them."""
import pytest
import torch

from nanorlhf_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_ref", [False, True])
def test_traced_losses_follow_their_inputs(with_ref):
    x, y, old, adv = (torch.randn(4, 300, device="cuda") * 0.3 for _ in range(4))
    mask = torch.rand(4, 300, device="cuda") > 0.3

    def policy(p):
        loss, stats = ops.policy_loss_token(p, old, adv, mask, 0.2, old + 0.1 if with_ref else None, 0.05 if with_ref else 0.0)
        return (loss, *stats.values())

    def value(p):
        return ops.value_loss(p, old, adv, mask, 0.2)
    for f in (policy, value):
        traced = torch.jit.trace(f, x, check_trace=False)
        for a, b in zip(traced(y), f(y)):
            assert torch.equal(a, b)
        p, q = (y.clone().requires_grad_(True) for _ in range(2))
        (2.0 * traced(p)[0]).backward()
        (2.0 * f(q)[0]).backward()
        assert torch.allclose(p.grad, q.grad, rtol=1e-6, atol=0)
