"""Float results of the general GEMM, stored and added to, at the edges of the rows and columns that a warp hands out together."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 3, 31, 33, 127, 130, 257])
@pytest.mark.parametrize("N", [8, 32, 40, 72, 264])
@pytest.mark.parametrize("a_mn", [False, True])
def test_float_results_and_sums(M, N, a_mn):
    from nanorlhf_b200.ops import gemm
    if a_mn and M % 8:
        M = (M + 7) // 8 * 8
    K = 136
    g = torch.Generator(device="cuda").manual_seed(M * N)
    a, b = (torch.randn(r, K, generator=g, device="cuda").bfloat16() for r in (M, N))
    want = 0.5 * a.double() @ b.double().T
    ops = (a.T.contiguous(), b.T.contiguous()) if a_mn else (a, b)
    wide = torch.full((M + 2, N + 8), 7.0, device="cuda")
    out = wide[1:M + 1, 4:N + 4]                             # rows of a larger tensor: nothing beside the result may change
    for accumulate, start in ((False, 0.0), (True, 7.0)):
        wide.fill_(7.0)
        gemm.gemm(*ops, a_mn=a_mn, b_mn=a_mn, alpha=0.5, out_f32=out, accumulate=accumulate)
        # products of 136 bf16 values, summed in float: a few 2^-24 of the terms' norm
        assert (out.double() - want - start).abs().max().item() < 1e-4
        edge = wide.clone()
        edge[1:M + 1, 4:N + 4] = 7.0
        assert torch.equal(edge, torch.full_like(edge, 7.0))
