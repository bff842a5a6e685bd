"""GEMMs whose contraction is cut into ranges on pairs of blocks, against float64: rows of the second block missing, columns that end inside a tile, ranges of
unequal length, sums by clusters and through a workspace, both forms of the second operand."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 128, 129, 257, 700])
@pytest.mark.parametrize("N", [72, 200, 1544])
@pytest.mark.parametrize("bn,splits,K", [(128, 2, 1032), (128, 4, 2112), (192, 2, 1032), (192, 3, 2112), (256, 2, 1032), (256, 4, 4168), (256, 7, 4168), (128, 8, 4168)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_against_float64(M, N, bn, splits, K, b_mn):
    from nanorlhf_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), generator=g, device="cuda").bfloat16()
    bias = torch.randn(N, generator=g, device="cuda").bfloat16()
    bt = b if b_mn else b.T
    ref = 0.5 * (a.double() @ bt.double()) + bias.double()
    mag = 0.5 * (a.double().abs() @ bt.double().abs()) + bias.double().abs()
    out = gemm.gemm(a, b, b_mn=b_mn, bias=bias, alpha=0.5, cg=2, block_n=bn, split_k=splits)
    # one rounding to bf16 and float sums of K products, cut off at 2^-23 of a partial sum every 16 products
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + K / 16 * 2.0 ** -23 * mag).all()
    for _ in range(3):                                       # ranges are added up in their order
        assert torch.equal(out, gemm.gemm(a, b, b_mn=b_mn, bias=bias, alpha=0.5, cg=2, block_n=bn, split_k=splits))


@pytest.mark.parametrize("M,N,K", [(1024, 1536, 8960), (512, 1536, 8960), (256, 3584, 18944), (770, 264, 65536)])
def test_taken_by_itself_and_on_two_streams(M, N, K):
    """A product on another stream has a workspace of its own."""
    from nanorlhf_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = torch.randn(M, K, generator=g, device="cuda").bfloat16(), torch.randn(N, K, generator=g, device="cuda").bfloat16()
    a2 = a.flip(0).contiguous()
    ref, ref2 = gemm.gemm(a, b), gemm.gemm(a2, b)
    want = a.double() @ b.double().T
    assert (ref.double() - want).norm() <= 2.0 ** -8 * want.norm()
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    outs = []
    for _ in range(4):
        for st, x in zip(s, (a, a2)):
            with torch.cuda.stream(st):
                outs.append(gemm.gemm(x, b))
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        assert torch.equal(o, ref if i % 2 == 0 else ref2)
