"""The log-probability head on pairs of blocks against float64: rows that end inside a pair's tile, vocabularies that end inside a tile, a chunk of 64 or a
range, one and several ranges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [129, 256, 505, 1030])
@pytest.mark.parametrize("V,ranges", [(72, 0), (250, 1), (257, 0), (1000, 3), (4104, 0), (4104, 16)])
def test_against_float64(M, V, ranges):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + V)
    K = 72
    h, w = torch.randn(M, K, generator=g, device="cuda").bfloat16(), (torch.randn(V, K, generator=g, device="cuda") * 0.3).bfloat16()
    t = torch.randint(0, V, (M,), generator=g, device="cuda").int()
    t[0], t[1], t[2] = 0, V - 1, min(V - 1, 64)
    logp, ent, lse = native.ext().lmhead_logprob_fwd(h, w, t, 1 / 0.9, ranges)
    z = h.double() @ w.double().T / 0.9
    lp = torch.log_softmax(z, -1)
    # logits as float sums of 72 products; exponentials and their sums to a few units of 2^-22
    tol = 2.0 ** -18 * (1 + z.abs().amax(1))
    assert ((logp.double() - lp.gather(1, t.long()[:, None])[:, 0]).abs() <= tol).all()
    assert ((lse.double() - torch.logsumexp(z, -1)).abs() <= tol).all()
    assert ((ent.double() + (lp.exp() * lp).sum(-1)).abs() <= 4 * tol).all()
