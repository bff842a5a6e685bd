"""SwiGLU of two projections in one GEMM: rows and features around its tiles, adapters of several ranks, and the calls it leaves alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,F,r", [(1, 64, 128, 0), (7, 1536, 520, 64), (256, 64, 128, 0), (300, 128, 200, 0), (257, 200, 136, 72), (513, 256, 392, 8), (1000, 1536, 8960, 64)])
def test_swiglu_linears_against_float64(M, K, F, r):
    from nanorlhf_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(M + F)

    def rnd(*shape):
        return (torch.randn(*shape, generator=g, device="cuda") * 0.1).bfloat16()
    x, weights = rnd(M, K) * 10, []
    want = []
    for _ in range(2):
        w, a, b = rnd(F, K), (rnd(r, K) if r else None), (rnd(F, r) if r else None)
        weights.append((w, a, b))
        y = x.double() @ w.double().T
        if r:
            y += 0.25 * (x.double() @ a.double().T) @ b.double().T
        want.append(y)
    want = torch.nn.functional.silu(want[0]) * want[1]
    got = gemm.swiglu_linears(x, *weights, scaling=0.25)
    # gate, up, the adapters' inner product and the result are rounded to bf16 (2^-9 at most, 1.7e-3 in the root mean square each): 3.3e-3 together
    assert ((got.double() - want).norm() / want.norm()).item() < 4e-3


def test_swiglu_linears_refusals_and_hooks():
    from nanorlhf_b200.models.lora import fused_swiglu_forward
    from nanorlhf_b200.models.qwen2 import Linear
    from nanorlhf_b200.ops import gemm
    w = torch.randn(128, 64, device="cuda").bfloat16()
    x = torch.randn(256, 64, device="cuda").bfloat16()
    assert gemm.swiglu_linears(x[:0], (w, None, None), (w, None, None)) is None
    assert gemm.swiglu_linears(x, (w, None, None), (w[:64], None, None)) is None
    gate, up = (Linear(64, 128, bias=False, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    assert fused_swiglu_forward(x, gate, up) is None          # autograd is on
    with torch.no_grad():
        assert fused_swiglu_forward(x, gate, up) is not None
        up.register_forward_hook(lambda *_: None)
        assert fused_swiglu_forward(x, gate, up) is None
