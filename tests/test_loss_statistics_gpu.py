"""The statistics that the losses return are the caller's: they may be changed in place, before the backward too."""
import pytest
import torch

from nanorlhf_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [50, 5000, 140000])          # one block, a cluster, many blocks
@pytest.mark.parametrize("value", [False, True])
def test_statistics_may_change_in_place(n, value):
    x, old, adv = (torch.randn(1, n, device="cuda") * 0.3 for _ in range(3))
    mask = torch.rand(1, n, device="cuda") > 0.3

    def run():
        p = x.clone().requires_grad_(True)
        if value:
            loss, frac = ops.value_loss(p, old, adv, mask, 0.2)
            return p, loss, {"clipfrac": frac}
        loss, stats = ops.policy_loss_token(p, old, adv, mask, 0.2, old + 0.1, 0.05)
        return p, loss, stats
    p, loss, stats = run()
    loss.backward()
    q, loss2, stats2 = run()
    want = {k: v.item() for k, v in stats2.items()}
    for i, v in enumerate(stats2.values()):
        assert not v._is_view() and v._version == 0 and not v.requires_grad
        v.mul_(i + 2.0)
    assert all(v.item() == pytest.approx(want[k] * (i + 2.0)) for i, (k, v) in enumerate(stats2.items()))      # none shares a value with another
    stats2["clipfrac"] += loss2                            # a statistic may take up a graph
    loss2.backward()
    assert torch.equal(p.grad, q.grad) and stats2["clipfrac"].requires_grad
