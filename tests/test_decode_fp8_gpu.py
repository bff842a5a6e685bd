"""Decode attention over fp8 pages, two pages a step: numbers of pages at which a warp's last step holds one page or two, or it has none, parts that end inside a
sequence, against float64 on the values that the pages hold."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv", [(12, 2), (28, 4), (3, 3), (8, 1)])
@pytest.mark.parametrize("splits", [1, 2, 5, 8])
def test_against_float64(Hq, Hkv, splits):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(Hq + splits)
    # one token; a page and a token more; pages of one, two, three and four steps of a warp (four warps, two pages a step) and their neighbours; page numbers beyond 32
    lens = [1, 16, 17, 63, 64, 65, 128, 129, 16 * 9, 16 * 12 + 5, 16 * 16, 16 * 17, 500, 16 * 4 * 32, 16 * 4 * 33 + 1]
    S, D, P = len(lens), 128, 16
    pages = [(n + P - 1) // P for n in lens]
    order, table, o = torch.randperm(sum(pages), generator=g, device="cuda").int(), torch.zeros(S, max(pages), dtype=torch.int32, device="cuda"), 0
    for i, n in enumerate(pages):
        table[i, :n] = order[o:o + n]
        o += n
    f8 = lambda *s: (torch.randn(*s, generator=g, device="cuda") * 100).clamp(-448, 448).to(torch.float8_e4m3fn)  # noqa: E731
    k, v = f8(sum(pages), Hkv, P, D), f8(sum(pages), Hkv, D, P)
    ks, vs = (torch.rand(sum(pages), Hkv, P, generator=g, device="cuda") * 0.01 + 0.005 for _ in range(2))
    q = torch.randn(S, Hq, D, generator=g, device="cuda").bfloat16()
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out = native.ext().paged_decode_fp8(q, k.view(torch.uint8), v.view(torch.uint8), ks, vs, table, ctx, 1 / math.sqrt(D), splits)
    kd, vd = k.double() * ks.double()[..., None], (v.double() * vs.double()[:, :, None]).transpose(2, 3)
    for i, n in enumerate(lens):
        kk, vv = (t[table[i, :pages[i]].long()].transpose(0, 1).reshape(Hkv, -1, D)[:, :n] for t in (kd, vd))
        p = torch.softmax(q[i].double().view(Hkv, -1, D) @ kk.transpose(1, 2) / math.sqrt(D), -1)
        want, mag = (p @ vv).reshape(Hq, D), (p @ vv.abs()).reshape(Hq, D)
        # weights to f16 (2^-11), the result to bf16 (2^-8), the rest in float
        assert ((out[i].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -10 * mag).all(), n
