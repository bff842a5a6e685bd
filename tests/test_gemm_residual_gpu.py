"""A residual added in a GEMM's epilogue: the bits of the product followed by the sum, on every tile, at ragged edges, with strides and cut contractions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _r(g, *s):
    return torch.randn(*s, generator=g, device="cuda").bfloat16()


@pytest.mark.parametrize("M,N", [(1, 8), (129, 72), (255, 200), (300, 264)])
@pytest.mark.parametrize("cg,bn", [(1, 64), (1, 128), (1, 192), (1, 256), (2, 128), (2, 192), (2, 256)])
def test_every_tile(M, N, cg, bn):
    from nanorlhf_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(M + N + cg + bn)
    a, b, res, bias = _r(g, M, 136), _r(g, N, 136), _r(g, M, N + 24)[:, 8:8 + N], _r(g, N)
    a2, b2 = _r(g, M, 16), _r(g, N, 16)
    kw = dict(a2=a2, b2=b2, bias=bias, alpha=0.5, cg=cg, block_n=bn)
    assert torch.equal(gemm.gemm(a, b, residual=res, **kw), gemm.gemm(a, b, **kw) + res)


@pytest.mark.parametrize("M,N,K", [(128, 512, 8960), (1000, 1536, 8960), (40, 64, 4096)])
def test_cut_contractions(M, N, K):
    from nanorlhf_b200.ops import gemm, native
    assert native.ext().gemm_tc_auto_splits(M, N, K) > 1
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b, res = _r(g, M, K), _r(g, N, K), _r(g, M, N)
    assert torch.equal(gemm.gemm(a, b, residual=res), gemm.gemm(a, b) + res)


@pytest.mark.parametrize("rank", [0, 8])
@pytest.mark.parametrize("train", [False, True])
def test_the_layers_mlp(rank, train):
    from nanorlhf_b200.models.lora import LoraLinear
    from nanorlhf_b200.models.qwen2 import Qwen2Config, Qwen2MLP
    torch.manual_seed(rank)
    mlp = Qwen2MLP(Qwen2Config(hidden_size=128, intermediate_size=264, num_attention_heads=1, num_key_value_heads=1)).cuda().bfloat16()
    if rank:
        for n in ("gate_proj", "up_proj", "down_proj"):
            setattr(mlp, n, LoraLinear(getattr(mlp, n), rank, 16))
            torch.nn.init.normal_(getattr(mlp, n).lora_B.weight, std=0.1)
    x, h, gy = (torch.randn(150, 128, device="cuda").bfloat16() for _ in range(3))

    def run(joint):
        xs, hs = x.clone().requires_grad_(train), h.clone().requires_grad_(train)
        with torch.set_grad_enabled(train):
            y = mlp(xs, hs) if joint else hs + mlp(xs)
        if not train:
            return [y]
        return [y, *torch.autograd.grad(y, [xs, hs, *[p for p in mlp.parameters() if p.requires_grad]], gy)]

    assert all(torch.equal(p, q) for p, q in zip(run(True), run(False)))
