"""Causal packed attention at the lengths where its tiles, key blocks and item order change, forward and backward, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = {
    "one": [1],
    "tile_edges": [127, 128, 129, 255, 256, 257, 1, 15, 16, 17],
    "long_short": [3, 1500, 64, 0, 777, 0, 1025],
    "many": [(7 * i) % 90 for i in range(70)],           # more sequences than lanes, some empty
    "ragged_items": [300 + 37 * i for i in range(40)],     # several items per CTA, levels that end at different sequences
}


@pytest.mark.parametrize("lens", LENS.values(), ids=LENS.keys())
@pytest.mark.parametrize("heads,kv_heads", [(4, 4), (6, 2), (7, 1)])
def test_attention_varlen_against_float64(lens, heads, kv_heads):
    from nanorlhf_b200.ops import native
    ext = native.ext()
    T, D = sum(lens), 128
    g = torch.Generator(device="cuda").manual_seed(T + heads)
    q, do = (torch.randn(T, heads, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(T, kv_heads, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    scale = 1 / math.sqrt(D)
    o, lse = ext.attn_fwd_tc(q, k, v, cu, scale)
    got = ext.attn_bwd_tc(do, q, k, v, o, lse, cu, scale)

    qd, kd, vd = (t.double().requires_grad_(True) for t in (q, k, v))
    outs, lses, t0 = [], [], 0
    for n in lens:
        qs, ks, vs = (t[t0:t0 + n].transpose(0, 1) for t in (qd, kd, vd))
        ks, vs = (t.repeat_interleave(heads // kv_heads, 0) for t in (ks, vs))
        s = (qs @ ks.transpose(1, 2) * scale).masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), -math.inf)
        outs.append((s.softmax(-1) @ vs).transpose(0, 1))
        lses.append(s.detach().logsumexp(-1))
        t0 += n
    want = torch.cat(outs)
    want.backward(do.double())

    def rel(a, b):
        return ((a.double() - b).norm() / b.norm().clamp_min(1e-6)).item()
    # P, dS and the results are rounded to bf16 (2^-9 each, independent); delta is formed from the rounded result
    assert rel(o, want.detach()) < 5e-3
    assert (lse.double() - torch.cat(lses, 1)).abs().max().item() < 1e-4
    if T > 1:
        for a, b in zip(got, (qd.grad, kd.grad, vd.grad)):
            assert rel(a, b) < 1e-2
