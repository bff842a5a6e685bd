"""GEMMs whose contraction is cut into ranges that a cluster sums through distributed shared memory (csrc/gemm_tc.cu): edges of tiles, ranges and clusters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 3, 5, 8])
@pytest.mark.parametrize("M,N,K", [(1, 8, 512), (129, 64, 1000), (127, 72, 4104), (300, 200, 576), (16, 1536, 1544), (640, 128, 2048)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_against_float64(M, N, K, a_mn, b_mn, splits):
    from nanorlhf_b200.ops import native
    if a_mn and M % 8:
        pytest.skip("rows of the operand are not on 16-byte boundaries")
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a = torch.randn(*((K, M) if a_mn else (M, K)), generator=g, device="cuda").bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), generator=g, device="cuda").bfloat16()
    bias = torch.randn(N, generator=g, device="cuda").bfloat16()
    run = lambda sp: native.ext().gemm_tc(a, b, a_mn, b_mn, None, None, bias, 0, 0.5, None, None, False, 0, 0, sp)  # noqa: E731
    got = run(splits)
    A, B = (a.T if a_mn else a).double(), (b if b_mn else b.T).double()
    want = 0.5 * (A @ B) + bias.double()
    # one rounding to bf16, and float sums of K products: 2^-24 sqrt(K) of the terms' norm, far below it
    bound = 2.0 ** -8 * want.abs() + K ** 0.5 * 2.0 ** -22 * (A.norm(dim=1)[:, None] * B.norm(dim=0)[None])
    assert ((got.double() - want).abs() <= bound).all()
    assert torch.equal(got, run(splits))


@pytest.mark.parametrize("K", [32768, 32832])                # the last pair of ranges that a cluster sums, the first through the workspace
@pytest.mark.parametrize("M,N", [(129, 72), (16, 64)])
def test_pairs_of_long_ranges_against_float64(M, N, K):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(K)
    a, b = (torch.randn(r, K, generator=g, device="cuda").bfloat16() for r in (M, N))
    run = lambda: native.ext().gemm_tc(a, b, False, False, None, None, None, 0, 0.5, None, None, False, 0, 0, 2)  # noqa: E731
    got, want = run(), 0.5 * (a.double() @ b.double().T)
    bound = 2.0 ** -8 * want.abs() + K ** 0.5 * 2.0 ** -22 * (a.double().norm(dim=1)[:, None] * b.double().norm(dim=1)[None])
    assert ((got.double() - want).abs() <= bound).all()
    assert torch.equal(got, run())
