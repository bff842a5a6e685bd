"""The warp-per-row norms at the widths where their forms change, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [8, 64, 1016, 1024, 1032, 1528, 1536, 1544, 2048, 2056, 3576, 3584, 3592, 8192])
@pytest.mark.parametrize("rows", [1, 5, 33])
def test_norms_against_float64(d, rows):
    from nanorlhf_b200.ops import native
    ext = native.ext()
    g = torch.Generator(device="cuda").manual_seed(d + rows)
    x, r, gy = (torch.randn(rows, d, generator=g, device="cuda").bfloat16() for _ in range(3))
    w, b = (torch.randn(d, generator=g, device="cuda").bfloat16() for _ in range(2))

    def rel(a, c):
        return ((a.double() - c).norm() / c.norm()).item()          # one rounding to bf16: 2^-9 at most per element, 1.7e-3 in norm

    def norm(t):
        return t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    s = (x.float() + r.float()).bfloat16()
    y, res, rstd = ext.rmsnorm(x, w, 1e-6, r, True)
    assert torch.equal(res, s) and rel(y, norm(s.double())) < 4e-3
    y, _, rstd = ext.rmsnorm(x, w, 1e-6, None, True)
    xd = x.double().requires_grad_(True)
    out = norm(xd)
    out.backward(gy.double())
    assert rel(y, out.detach()) < 4e-3 and rel(ext.rmsnorm_bwd(x, w, gy, rstd), xd.grad) < 4e-3
    if d <= 2048:
        for rr in (r, None):
            t = x.double() + (r.double() if rr is not None else 0.0)
            want = torch.nn.functional.layer_norm(t, (d,), w.double(), b.double(), 1e-7)
            assert rel(ext.add_layernorm(x, rr, w, b, 1e-7), want) < 4e-3
