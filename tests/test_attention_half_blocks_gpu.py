"""Packed causal attention where the last block of a sequence holds about half of its keys: the other half is left out."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[63], [64], [65], [192, 193, 191, 1], [320, 64, 0, 449, 448], [64] * 40, [65] * 40])
def test_ends_of_sequences_against_float64(lens):
    from nanorlhf_b200.ops import native
    T, H, K, D = sum(lens), 6, 2, 128
    g = torch.Generator(device="cuda").manual_seed(T)
    q = torch.randn(T, H, D, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(T, K, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    o, lse = native.ext().attn_fwd_tc(q, k, v, cu, 1 / math.sqrt(D))
    t0 = 0
    for n in lens:
        if n == 0:
            continue
        qs, ks, vs = (t[t0:t0 + n].double().transpose(0, 1) for t in (q, k, v))
        ks, vs = (t.repeat_interleave(H // K, 0) for t in (ks, vs))
        s = (qs @ ks.transpose(1, 2) / math.sqrt(D)).masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), -math.inf)
        want = (s.softmax(-1) @ vs).transpose(0, 1)
        # P and the result are rounded to bf16 (2^-9 each)
        assert ((o[t0:t0 + n].double() - want).norm() / want.norm()).item() < 5e-3
        assert (lse[:, t0:t0 + n].double() - s.logsumexp(-1)).abs().max().item() < 1e-4
        t0 += n
