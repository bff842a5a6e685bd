"""The cluster sampler's nucleus rule and its copy pieces at the sizes where they change, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [8, 4096, 8192, 8200, 8192 * 2 + 8, 51200, 51208, 151936])      # one vector; a piece and one more; 1, 2 and 4 slices
@pytest.mark.parametrize("kind", ["flat", "tied", "masked"])
def test_drawn_tokens_lie_in_the_nucleus(V, kind):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(V)
    z = torch.randn(64, V, generator=g, device="cuda") * 2
    if kind == "tied":
        z = z.round()                                        # a handful of values: whole classes of equal tokens
    if kind == "masked":
        z[:, 1:] = torch.where(torch.rand(64, V - 1, generator=g, device="cuda") < 0.5, torch.full_like(z[:, 1:], -float("inf")), z[:, 1:])
    z = z.bfloat16()
    tok = torch.stack([native.sample(z, 0.9, 0.8, 5, s, impl=2) for s in range(8)], 1).long()
    p = torch.softmax(z.double() / 0.9, -1)
    for c in range(8):
        mine = z.gather(1, tok[:, c:c + 1])
        above = (p * (z > mine)).sum(1)
        assert (p.gather(1, tok[:, c:c + 1]) > 0).all()
        assert (above < 0.8 + 1e-5).all()                    # float32 sums of V terms against float64
    assert torch.equal(tok[:, 0], native.sample(z, 0.9, 0.8, 5, 0, impl=2).long())
