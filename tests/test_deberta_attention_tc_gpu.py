"""Disentangled attention on tcgen05 (csrc/attention_deberta_tc.cu) against float64, at the edges of its tiles (128 queries, 64 keys, 64 buckets)."""
import math

import pytest
import torch

from nanorlhf_b200.models.deberta_v3 import build_bucket_lut

pytestmark = pytest.mark.gpu


def _inputs(lens, heads, buckets, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T = sum(lens)
    qkv = torch.randn(T, 3, heads, 64, generator=g, device="cuda").bfloat16()
    pos_k, pos_q = (torch.randn(buckets, heads, 64, generator=g, device="cuda").bfloat16().transpose(0, 1) for _ in range(2))
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    return [qkv[:, i].contiguous() for i in range(3)], pos_k, pos_q, cu


def _reference(qkv, pos_k, rel_b, lut, lens, scale):
    q, k, v = (t.double().transpose(0, 1) for t in qkv)
    rel_a = torch.bmm(q.float(), pos_k.float().transpose(1, 2)).bfloat16().double()          # rounded as the kernel rounds it
    out, s0, center = [], 0, (lut.numel() - 1) // 2
    for n in lens:
        i, r = torch.arange(n, device="cuda"), slice(s0, s0 + n)
        c = lut.long()[i[:, None] - i[None, :] + center][None].expand(q.shape[0], n, n)
        s = q[:, r] @ k[:, r].transpose(1, 2) + rel_a[:, r].gather(2, c) + rel_b[:, r].double().gather(2, c.transpose(1, 2)).transpose(1, 2)
        out.append((torch.softmax(s * scale, -1) @ v[:, r]).transpose(0, 1))
        s0 += n
    return torch.cat(out)


@pytest.mark.parametrize("lens,heads,span,top", [
    ([1], 16, 256, 512), ([64], 2, 256, 512), ([65], 1, 256, 512), ([128, 129, 1, 63], 3, 256, 512), ([700, 40, 1], 2, 256, 512),
    ([1663, 640, 641], 2, 256, 512),                 # blocks with one bucket for all differences
    ([1300], 2, 16, 64), ([500, 90], 2, 4, 16),      # few buckets, far fewer than the 144 columns of a window
    ([900], 2, 100, 4000),                           # a bucket that still changes at the far end
    ([2, 3] * 40, 16, 256, 512),                     # more items than SMs
])
def test_against_float64(lens, heads, span, top):
    from nanorlhf_b200.models.deberta_v3 import _bias_tables
    from nanorlhf_b200.ops import native
    qkv, pos_k, pos_q, cu = _inputs(lens, heads, 2 * span)
    lut = build_bucket_lut(max(lens), span, top, span, "cuda")
    rel_b, scale = _bias_tables(qkv[1], pos_q), 1.0 / math.sqrt(192)
    got = native.ext().deberta_attn_tc(*qkv, cu, max(lens), scale, pos_k, rel_b, lut)
    want = _reference(qkv, pos_k, rel_b, lut, lens, scale)
    # weights and results are rounded to bf16 once each: 2^-9 of every term and 2^-9 of the result.  A sum of A on the other side of a rounding boundary
    # moves its score by 2^-8 |A| scale and one weight by that factor: below 2^-8 for |A| up to 14, six standard deviations being 48, so one in many
    assert torch.isfinite(got).all()
    assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert (got.double() - want).abs().max() <= 2.0 ** -7 * (qkv[2].double().abs().max() + want.abs().max())
    assert torch.equal(got, native.ext().deberta_attn_tc(*qkv, cu, max(lens), scale, pos_k, rel_b, lut))


@pytest.mark.parametrize("lens", [[300, 129], [40], [64]])
def test_large_scores(lens):
    """Scores of 2^17 and more in front of the softmax, a different size in every row: what is subtracted from them has to be as exact as they are."""
    from nanorlhf_b200.models.deberta_v3 import _bias_tables
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(2)
    T, heads, buckets, scale = sum(lens), 2, 512, 0.75
    small = lambda *shape: torch.randint(-2, 3, shape, generator=g, device="cuda").to(torch.bfloat16) / 2  # noqa: E731
    q, k, v = small(T, heads, 64), small(T, heads, 64), torch.randn(T, heads, 64, generator=g, device="cuda").bfloat16()
    pos_k, pos_q = (small(buckets, heads, 64).transpose(0, 1) for _ in range(2))
    q[:, :, 0], k[:, :, 0] = 256.0 + 2.0 * torch.arange(T, device="cuda")[:, None] % 200, 512.0
    pos_k[:, :, 0], pos_q[:, :, 0] = 0.0, 0.0
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    lut = build_bucket_lut(max(lens), 256, 512, 256, "cuda")
    rel_b = _bias_tables(k, pos_q)
    got = native.ext().deberta_attn_tc(q, k, v, cu, max(lens), scale, pos_k, rel_b, lut)
    want = _reference([q, k, v], pos_k, rel_b, lut, lens, scale)
    # every product is a multiple of a quarter and every sum below 2^18, so that scores are exact; scaled they are rounded to 2^-7 once, the same for all keys
    assert torch.isfinite(got).all()
    assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("std", [0.5, 1.0, 1.5, 2.0])           # of the operands: flat rows to single weights
@pytest.mark.parametrize("lens", [[1536], [300, 300], [40] * 8, [700, 90]])
def test_no_further_from_float64_than_the_kernel_with_two_tables(lens, std):
    from nanorlhf_b200.models.deberta_v3 import _bias_tables
    from nanorlhf_b200.ops import native
    (q, k, v), pos_k, pos_q, cu = _inputs(lens, 8, 512, seed=4)
    q, k, pos_k, pos_q = ((t.float() * std).bfloat16() for t in (q, k, pos_k.transpose(0, 1), pos_q.transpose(0, 1)))
    pos_k, pos_q = pos_k.transpose(0, 1), pos_q.transpose(0, 1)
    lut, scale = build_bucket_lut(max(lens), 256, 512, 256, "cuda"), 1.0 / math.sqrt(192)
    rel_b = _bias_tables(k, pos_q)
    want = _reference([q, k, v], pos_k, rel_b, lut, lens, scale)
    new = native.ext().deberta_attn_tc(q, k, v, cu, max(lens), scale, pos_k, rel_b, lut)
    old = native.ext().deberta_attn_fwd(q, k, v, cu, max(lens), scale, _bias_tables(q, pos_k), rel_b, lut)
    # both round each weight and each result once, a row's largest weight being 1; how often it is another block's that is rounded differs by a share of
    # a per cent either way, and so does the rounding of A
    assert (new.double() - want).norm() <= 1.005 * (old.double() - want).norm()


def test_rows_of_a_wider_projection_and_tables():
    """q, k and v as columns of one product, against the kernel that reads both tables."""
    from nanorlhf_b200.models.deberta_v3 import _bias_tables
    from nanorlhf_b200.ops import native
    lens, heads = [300, 77], 4
    qkv, pos_k, pos_q, cu = _inputs(lens, heads, 512, seed=1)
    lut = build_bucket_lut(300, 256, 512, 256, "cuda")
    wide = torch.cat([t.reshape(-1, heads * 64) for t in qkv], 1)
    q, k, v = (wide[:, i * heads * 64:(i + 1) * heads * 64].unflatten(1, (heads, 64)) for i in range(3))
    got = native.ext().deberta_attn_tc(q, k, v, cu, 300, 0.07, pos_k, _bias_tables(k, pos_q), lut)
    old = native.ext().deberta_attn_fwd(q, k, v, cu, 300, 0.07, _bias_tables(q, pos_k), _bias_tables(k, pos_q), lut)
    assert (got.float() - old.float()).norm() <= 2.0 ** -8 * old.float().norm()
    with pytest.raises(RuntimeError):
        native.ext().deberta_attn_tc(q, k, v, cu, 301 + 64, 0.07, pos_k, _bias_tables(k, pos_q), lut)
