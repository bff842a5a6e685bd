"""The loss kernels and the advantage scan at the sizes where their forms change, against float64."""
import pytest
import torch

from nanorlhf_b200 import ops
from nanorlhf_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30)).item()


@pytest.mark.parametrize("T", [1, 7, 8, 9, 256, 2047, 2048, 2049, 4097])      # a thread's steps, a warp's, one tile and one step more
@pytest.mark.parametrize("gamma,lam", [(1.0, 0.95), (0.9, 0.5), (1.0, 1.0)])
def test_gae_against_float64(T, gamma, lam):
    g = torch.Generator(device="cuda").manual_seed(T)
    r, v = (torch.randn(3, T, generator=g, device="cuda") for _ in range(2))
    adv, ret = ops.gae(r, v, gamma, lam)
    a64, r64 = ref.gae(r.double(), v.double(), gamma, lam)
    # each sum rounds at most T times, errors add like a random walk: sqrt(4097) 2^-24 is 4e-6
    assert _rel(adv, a64) < 4e-6 and _rel(ret, r64) < 4e-6
    assert _rel(ops.discounted_suffix_sum(r, gamma), ref.discounted_suffix_sum(r.double(), gamma)) < 4e-6


@pytest.mark.parametrize("n", [1, 1024, 1025, 4097, 131072, 131073])          # one block, clusters of 2 and 8, the largest cluster, many blocks
@pytest.mark.parametrize("with_ref", [False, True])
def test_losses_against_float64(n, with_ref):
    g = torch.Generator(device="cuda").manual_seed(n)
    f = lambda s: torch.randn(1, n, generator=g, device="cuda") * s  # noqa: E731
    new, old, adv = f(0.5), f(0.5), f(1.0)
    refl, kl = (f(0.5), 0.05) if with_ref else (None, 0.0)
    mask = torch.rand(1, n, generator=g, device="cuda") > 0.3
    mask[0, 0] = True
    x, y = new.clone().requires_grad_(True), new.double().requires_grad_(True)
    loss, st = ops.policy_loss_token(x, old, adv, mask, 0.2, refl, kl)
    want, st64 = ref.policy_loss_token(y, old.double(), adv.double(), mask, 0.2, None if refl is None else refl.double(), kl)
    (3.0 * loss).backward()
    (3.0 * want).backward()
    # __expf is good to a few 2^-22 here and losses cancel between signs of the advantage: absolute against terms of order one
    assert abs(loss.item() - want.item()) < 4e-6 and _rel(x.grad, y.grad) < 2e-6
    assert set(st) == set(st64) and all(abs(st[k].item() - st64[k].item()) < 4e-6 for k in st64 if k != "clipfrac")
    assert abs(st["clipfrac"].item() - st64["clipfrac"].item()) <= 2.0 / n + 1e-6      # a ratio on the clip's edge may round either way
    x, y = f(1.0), f(1.0)
    v, w = x.clone().requires_grad_(True), x.double().requires_grad_(True)
    vl, cf = ops.value_loss(v, y, adv, mask, 0.2)
    vw, cw = ref.value_loss(w, y.double(), adv.double(), mask, 0.2)
    vl.backward()
    vw.backward()
    assert _rel(vl, vw) < 2e-6 and _rel(v.grad, w.grad) < 2e-6 and abs(cf.item() - cw.item()) <= 2.0 / n + 1e-6


def test_loss_gradient_can_carry_a_graph():
    x = torch.randn(1, 50, device="cuda", requires_grad=True)
    s = torch.ones((), device="cuda", requires_grad=True)
    loss, _ = ops.policy_loss_token(x, x.detach() + 0.1, torch.randn(1, 50, device="cuda"), torch.ones(1, 50, dtype=torch.bool, device="cuda"), 0.2)
    (g,) = torch.autograd.grad(loss * s, x, create_graph=True)
    (gs,) = torch.autograd.grad(g.sum(), s)
    assert torch.allclose(gs, g.detach().sum())
