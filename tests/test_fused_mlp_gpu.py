"""The training step's fused GEMMs against float64: sums of products in one accumulator, gate and up kept beside their product, and the product's gradient
taken apart in the epilogue; at the edges of tiles, slabs (32 x 64) and contraction blocks (64)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HALF = 2.0 ** -8            # rounding to bf16 (eight bits), relative
SUM = 2.0 ** -20            # float sums over at most 600 products, relative to the sum of their magnitudes (the tensor cores cut off: 2^-23 a step of 16)


def _r(g, *shape, std=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * std).bfloat16()


@pytest.mark.parametrize("M", [1, 255, 257, 1300])
@pytest.mark.parametrize("N", [8, 200, 1544])
@pytest.mark.parametrize("Ks", [(8,), (64, 200), (72, 8, 136, 64)])
def test_sum_of_products(M, N, Ks):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M * N + len(Ks))
    a, b = [_r(g, M, k) for k in Ks], [_r(g, k, N) for k in Ks]
    wide = _r(g, M, Ks[0] + 16)                               # one operand with rows of its own stride
    a[0] = wide[:, 8:8 + Ks[0]]
    ref = sum(x.double() @ y.double() for x, y in zip(a, b))
    mag = sum(x.double().abs() @ y.double().abs() for x, y in zip(a, b))
    out = native.ext().gemm_tc_sum(a, b)
    assert ((out.double() - ref).abs() <= HALF * 1.01 * ref.abs() + SUM * mag).all()


@pytest.mark.parametrize("M,F,K,r", [(1, 8, 8, 8), (33, 56, 64, 8), (256, 264, 72, 64), (300, 520, 200, 16)])
def test_gate_and_up_kept(M, F, K, r):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + F)
    x, wg, wu, t, bg, bu = _r(g, M, K), _r(g, F, K, std=K ** -0.5), _r(g, F, K, std=K ** -0.5), _r(g, M, 2 * r), _r(g, F, r, std=0.1), _r(g, F, r, std=0.1)
    act, gate, up = native.ext().gemm_tc_swiglu_pair_keep(x, wg, wu, t[:, :r], t[:, r:], bg, bu)
    for y, w, tt, b in ((gate, wg, t[:, :r], bg), (up, wu, t[:, r:], bu)):
        ref = x.double() @ w.double().T + tt.double() @ b.double().T
        mag = x.double().abs() @ w.double().abs().T + tt.double().abs() @ b.double().abs().T
        assert ((y.double() - ref).abs() <= HALF * 1.01 * ref.abs() + SUM * mag).all()
    assert torch.equal(act, native.ext().gemm_tc_swiglu_pair(x, wg, wu, t[:, :r], t[:, r:], bg, bu))
    ref = torch.nn.functional.silu(gate.double()) * up.double()
    assert ((act.double() - ref).abs() <= HALF * 1.01 * ref.abs() + 1e-30).all()


@pytest.mark.parametrize("M,F,K,r", [(1, 8, 8, 8), (32, 64, 64, 8), (33, 72, 56, 16), (257, 264, 136, 64), (700, 1544, 520, 64)])
def test_gradients_of_gate_and_up(M, F, K, r):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + F + K)
    dy, w, t, a = _r(g, M, K), _r(g, K, F, std=K ** -0.5), _r(g, M, r), _r(g, r, F, std=0.1)
    gate, up = _r(g, M, F, std=2.0), _r(g, M, F, std=2.0)
    dg, du = native.ext().gemm_tc_dswiglu(dy, w, t, a, gate, up)
    d = dy.double() @ w.double() + t.double() @ a.double()
    mag = dy.double().abs() @ w.double().abs() + t.double().abs() @ a.double().abs()
    gd, ud, s = gate.double(), up.double(), torch.sigmoid(gate.double())
    for got, f in ((dg, ud * (s + gd * s * (1 - s))), (du, gd * s)):
        # the gradient of the product is rounded to bf16, and so is the result; s + g s (1 - s) can cancel: float, 2^-20 of its terms
        err = 2.02 * HALF * (d * f).abs() + SUM * mag * f.abs() + 2.0 ** -20 * d.abs() * (ud.abs() + gd.abs()) * (1 + gd.abs())
        assert ((got.double() - d * f).abs() <= err + 1e-30).all()


def _mlp(seed=0):
    from nanorlhf_b200.models.lora import LoraConfig, get_peft_model
    from nanorlhf_b200.models.qwen2 import Qwen2Config, Qwen2ForCausalLM
    cfg = Qwen2Config.tiny()
    model = get_peft_model(Qwen2ForCausalLM.from_config(cfg, torch.bfloat16, "cuda", seed=seed), LoraConfig(r=8, lora_alpha=16))
    mlp = model.base_model.model.layers[0].mlp
    g = torch.Generator(device="cuda").manual_seed(5)
    with torch.no_grad():
        for n, p in mlp.named_parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") * (0.1 if "lora_A" not in n else 0.2))
    return mlp, cfg.hidden_size


@pytest.mark.parametrize("T", [1, 77, 1200])
@pytest.mark.parametrize("need_x", [True, False])
def test_module_takes_the_fused_form_and_a_hook_takes_it_apart(T, need_x):
    mlp, d = _mlp()
    g = torch.Generator(device="cuda").manual_seed(T)
    x, gy = _r(g, T, d).requires_grad_(need_x), _r(g, T, d)
    params = [p for p in mlp.parameters() if p.requires_grad]

    def run():
        y = mlp(x)
        return y, y.grad_fn.name(), torch.autograd.grad(y, ([x] if need_x else []) + params, gy)

    y, name, grads = run()
    assert "LoraMlp" in name
    seen = []
    h = mlp.gate_proj.register_forward_pre_hook(lambda m, a: seen.append(1))
    y2, name2, grads2 = run()
    h.remove()
    assert "LoraMlp" not in name2
    assert torch.equal(y, y2)
    for a, b in zip(grads, grads2):
        # the sum over gate and up is rounded once instead of three times, products in another order: a few bf16 roundings
        assert (a.double() - b.double()).norm() <= 2 * HALF * b.double().norm()
