"""Gradient of the log-probability head's logits at the row counts where it changes between single CTAs and CTA pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 127, 128, 129, 256, 257, 300, 384, 385, 512, 513, 640, 896, 897])
@pytest.mark.parametrize("V,K", [(1000, 64), (4104, 200)])
def test_dlogits_against_float64(M, V, K):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + V)
    h = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(V, K, generator=g, device="cuda") * 0.2).bfloat16()
    t = torch.randint(0, V, (M,), generator=g, device="cuda", dtype=torch.int32)
    grad = torch.randn(M, generator=g, device="cuda")
    inv_t = 1 / 0.9
    z = h.double() @ w.double().T * inv_t
    lse = z.logsumexp(-1)
    want = (torch.nn.functional.one_hot(t.long(), V).double() - (z - lse[:, None]).exp()) * (grad.double() * inv_t)[:, None]
    got = native.ext().lmhead_dlogits(h, w, t, lse.float(), grad, inv_t)
    # rounded to bf16 once (2^-9 at most per element)
    assert ((got.double() - want).norm() / want.norm()).item() < 4e-3
