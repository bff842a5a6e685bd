"""The head's statistics from one range of the vocabulary per SM: last rows of a block that combines them, fewer and more ranges than its threads a row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,ranges", [(1, 148), (31, 7), (33, 148), (128, 0), (128, 9), (256, 0), (256, 74), (300, 49)])
def test_against_float64(M, ranges):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + ranges)
    V, K = 37896, 72
    h, w = torch.randn(M, K, generator=g, device="cuda").bfloat16(), (torch.randn(V, K, generator=g, device="cuda") * 0.3).bfloat16()
    t = torch.randint(0, V, (M,), generator=g, device="cuda").int()
    t[-1] = V - 1
    logp, ent, lse = native.ext().lmhead_logprob_fwd(h, w, t, 1 / 0.9, ranges)
    z = h.double() @ w.double().T / 0.9
    lp = torch.log_softmax(z, -1)
    # logits as float sums of 72 products; exponentials and their sums to a few units of 2^-22
    tol = 2.0 ** -18 * (1 + z.abs().amax(1))
    assert ((logp.double() - lp.gather(1, t.long()[:, None])[:, 0]).abs() <= tol).all()
    assert ((lse.double() - torch.logsumexp(z, -1)).abs() <= tol).all()
    assert ((ent.double() + (lp.exp() * lp).sum(-1)).abs() <= 4 * tol).all()
