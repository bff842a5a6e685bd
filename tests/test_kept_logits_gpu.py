"""The head's logits kept for its backward: what is stored, the gradient formed from it and the calls that keep nothing."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _head(M, V, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, w = torch.randn(M, K, generator=g, device="cuda").bfloat16(), (torch.randn(V, K, generator=g, device="cuda") * 0.3).bfloat16()
    t = torch.randint(0, V, (M,), generator=g, device="cuda")
    t[0], t[-1] = V - 1, 0
    return h, w, t, torch.randn(M, generator=g, device="cuda")


@pytest.mark.parametrize("M", [1, 128, 129, 256, 300, 513])                  # both kernels, their last rows
@pytest.mark.parametrize("V", [8, 264, 8200, 16392])                         # the last columns of tiles and of a block's share of the gradient
def test_stored_logits_and_their_gradient(M, V):
    from nanorlhf_b200.ops import native
    ext = native.ext()
    h, w, t, g = _head(M, V, 72, M + V)
    z = torch.full((M + 1, V), 7.0, device="cuda")
    t32 = t.int()
    plain = ext.lmhead_logprob_fwd(h, w, t32, 1 / 0.9, 0)
    kept = ext.lmhead_logprob_fwd(h, w, t32, 1 / 0.9, 0, z[:M])
    assert all(torch.equal(a, b) for a, b in zip(plain, kept)) and (z[M] == 7.0).all()
    want, mag = h.double() @ w.double().T, h.double().abs() @ w.double().abs().T
    assert ((z[:M].double() - want).abs() <= 16 * 2.0 ** -23 * mag).all()     # float sums of 72 products, before the temperature
    lse = kept[2]
    assert torch.equal(ext.logits_grad(z[:M], t32, lse, g, 1 / 0.9), ext.lmhead_dlogits(h, w, t32, lse, g, 1 / 0.9))


@pytest.mark.parametrize("M,V", [(37, 1000), (300, 4096)])
def test_gradients_are_those_of_the_second_product(M, V):
    from nanorlhf_b200 import ops
    h, w, t, g = _head(M, V, 136, M)

    def grads(hooks, twice=False):
        x, y = h.clone().requires_grad_(), w.clone().requires_grad_()
        if hooks:
            with torch.autograd.graph.saved_tensors_hooks(lambda s: s, lambda s: s):
                lp, _ = ops.lmhead_logprob(x, y, t, 0.9, True)
        else:
            lp, _ = ops.lmhead_logprob(x, y, t, 0.9, True)
        if twice:
            torch.autograd.grad(lp, (x, y), g, retain_graph=True)
        return torch.autograd.grad(lp, (x, y), g)

    want = grads(True)
    for got in (grads(False), grads(False, True)):
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_what_keeps_nothing():
    from nanorlhf_b200.ops import native
    ext = native.ext()
    h = torch.empty(65536, 8, dtype=torch.bfloat16, device="cuda")
    assert ext.lmhead_logits_buffer(h[:1000], 1024).shape == (1000, 1024)
    assert ext.lmhead_logits_buffer(h, 16392) is None and ext.lmhead_logits_buffer(h[:5], 1004) is None and ext.lmhead_logits_buffer(h[:0], 1024) is None
    with torch.autograd.graph.saved_tensors_hooks(lambda s: s, lambda s: s):
        assert ext.lmhead_logits_buffer(h[:1000], 1024) is None
    before = torch.cuda.memory_allocated()
    with torch.no_grad():
        native.lmhead_logprob(h[:1024], torch.empty(1024, 8, dtype=torch.bfloat16, device="cuda", requires_grad=False), torch.zeros(1024, device="cuda", dtype=torch.long))
    assert torch.cuda.memory_allocated() == before
