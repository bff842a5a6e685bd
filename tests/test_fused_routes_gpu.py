"""The decoder's calls outside autograd on the GPU: what they give there is what the same calls give under autograd, tracing and transforms."""
import pytest
import torch

from nanorlhf_b200.models.qwen2 import Qwen2Config, Qwen2ForCausalLM

pytestmark = pytest.mark.gpu


def _mlp(width=256, ff=512):
    cfg = Qwen2Config(vocab_size=256, num_hidden_layers=1, hidden_size=width, intermediate_size=ff, num_attention_heads=2, num_key_value_heads=1,
                      head_dim=128)
    return Qwen2ForCausalLM.from_config(cfg, torch.bfloat16, "cuda", seed=0).model.layers[0].mlp


def test_a_traced_mlp_follows_its_inputs():
    mlp = _mlp()
    x, y = (torch.randn(300, 256, device="cuda").bfloat16() for _ in range(2))
    with torch.no_grad():
        traced = torch.jit.trace(mlp, x, check_trace=False)
        assert torch.allclose(traced(y).float(), mlp(y).float(), rtol=1e-2, atol=1e-2 * mlp(y).abs().max().item())      # one rounding apart at most


def test_forward_mode_is_refused_and_loses_no_tangent():
    mlp, fw = _mlp(), torch.autograd.forward_ad
    x = torch.randn(300, 256, device="cuda").bfloat16()
    with torch.no_grad(), fw.dual_level(), pytest.raises(NotImplementedError):
        mlp(fw.make_dual(x, x))


@pytest.mark.parametrize("rows", [1, 100, 128, 129, 257, 1000])
@pytest.mark.parametrize("K,F,r", [(1536, 8960, 64), (256, 520, 8), (1536, 8960, 0), (4096, 1024, 0), (200, 136, 0)])
def test_swiglu_rounds_alike_with_and_without_autograd(rows, K, F, r):
    from nanorlhf_b200 import ops
    from nanorlhf_b200.models.lora import LoraLinear, fused_swiglu_forward, lora_group_forward
    from nanorlhf_b200.models.qwen2 import Linear
    g = torch.Generator(device="cuda").manual_seed(rows + F)
    pair = [Linear(K, F, bias=False, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    if r:
        pair = [LoraLinear(m, r, 16) for m in pair]
        for m in pair:
            torch.nn.init.normal_(m.lora_B.weight, std=0.05, generator=g)
    x = torch.randn(rows, K, generator=g, device="cuda").bfloat16()
    want = ops.swiglu_pair(*lora_group_forward(x.requires_grad_(True), pair)).detach()
    with torch.no_grad():
        got = fused_swiglu_forward(x, *pair)
    if r or rows > 1152:
        assert got is not None
    assert got is None or torch.equal(got, want)


@pytest.mark.parametrize("adapters", [False, True])
@pytest.mark.parametrize("lens", [[37], [300, 1, 211], [1500, 700]])
def test_log_probabilities_of_an_unchanged_policy_do_not_move(adapters, lens):
    """Layers and head as the log-probability pass and the training forward run them: the ratio of the policy to itself is 1."""
    from nanorlhf_b200 import ops
    from nanorlhf_b200.models.lora import LoraConfig, get_peft_model
    cfg = Qwen2Config(vocab_size=1024, num_hidden_layers=3, hidden_size=512, intermediate_size=2048, num_attention_heads=4, num_key_value_heads=2,
                      head_dim=128)
    model = Qwen2ForCausalLM.from_config(cfg, torch.bfloat16, "cuda", seed=0)
    if adapters:
        model = get_peft_model(model, LoraConfig(r=64, lora_alpha=16))
        for n, p in model.named_parameters():
            if "lora_B" in n:
                torch.nn.init.normal_(p, std=0.02)
    base = model.base_model if adapters else model
    T = sum(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    cos, sin = ops.ref.rope_cos_sin(torch.cat([torch.arange(n, device="cuda") for n in lens]), 128, 1e6)
    x0 = torch.randn(T, 512, device="cuda").bfloat16()
    target = torch.randint(0, 1024, (T,), device="cuda")
    weight = torch.randn(1024, 512, device="cuda").bfloat16() * 0.05

    def logp(x):
        for layer in base.model.layers:
            x = layer(x, cos, sin, cu, max(lens))
        return ops.lmhead_logprob(x, weight, target, 0.9)[0]
    with torch.no_grad():
        old = logp(x0)
    assert torch.equal(old, logp(x0.clone().requires_grad_(True)).detach())
