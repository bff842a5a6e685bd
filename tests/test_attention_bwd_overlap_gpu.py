"""Gradients of training attention, whose kernels and readers overlap on the stream (csrc/attention_bwd_tc.cu): every one sees this pass's values, also
where an earlier pass left others at the same addresses."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, do, lens):
    """dQ, dK and dV in float64."""
    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    group, s0, out = q.shape[1] // k.shape[1], 0, []
    for n in lens:
        r = slice(s0, s0 + n)
        kr, vr = (t[r].repeat_interleave(group, 1).transpose(0, 1) for t in (k, v))
        s = q[r].transpose(0, 1) @ kr.transpose(1, 2) / math.sqrt(q.shape[2])
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), -math.inf)
        out.append((torch.softmax(s, -1) @ vr).transpose(0, 1))
        s0 += n
    return torch.autograd.grad(torch.cat(out), (q, k, v), do.double())


@pytest.mark.parametrize("lens,heads,kv", [([1], 12, 2), ([700, 130], 12, 2), ([64] * 9, 28, 4), ([3000], 12, 2), ([1500, 40, 900], 28, 4)])
def test_readers_behind_the_backward_see_all_gradients(lens, heads, kv):
    from nanorlhf_b200 import ops
    from nanorlhf_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(0)
    T = sum(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    sets = [[torch.randn(T, h, 128, generator=g, device="cuda").bfloat16() for h in (heads, kv, kv, heads)] for _ in range(3)]
    q, k, v, do = (torch.empty_like(t) for t in sets[0])
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    w = torch.randn(kv * 128, kv * 128, generator=g, device="cuda").bfloat16()
    sizes = [heads * T, T * heads * 64, T * kv * 64, T * kv * 64]          # delta, dQ, dK and dV, in floats

    def run(n):
        with torch.no_grad():
            for dst, src in zip((q, k, v, do), sets[n]):                   # other values at the same addresses
                dst.copy_(src)
        o = ops.attention_varlen(*leaves, cu, max(lens))
        spoilt = [torch.full((m,), math.nan, device="cuda") for m in sizes for _ in range(2)]
        del spoilt                                                         # what the backward allocates begins as NaN
        dq, dk, dv = torch.autograd.grad(o, leaves, do)
        # readers at once, one of them launched over the end of the backward, and buffers that take the place of freed ones
        return gemm.gemm(dk.view(T, -1), w), dv.clone(), dq.clone(), dk

    firsts = []
    for n in range(3):
        first = run(n)
        torch.cuda.synchronize()
        want_q, want_k, want_v = _reference(*sets[n], lens)
        for got, want in zip(first[1:], (want_v, want_q, want_k)):
            # O, P, dS and the result are rounded to bf16 once each, 2^-9; gradients that cancel are left with the rounding of delta's 128 products
            assert (got.double() - want).norm() <= 2.0 ** -7 * want.norm() + 2.0 ** -12 * got.numel() ** 0.5
        product = first[3].view(T, -1).double() @ w.double().T
        assert (first[0].double() - product).norm() <= 2.0 ** -8 * product.norm()
        firsts.append(first)
    runs = [(n, run(n)) for n in [0, 1, 2, 1, 0, 2] * 3]                   # nothing is waited for in between
    torch.cuda.synchronize()
    for n, again in runs:
        assert all(torch.equal(a, b) for a, b in zip(firsts[n], again))
