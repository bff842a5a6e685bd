"""What is timed when this framework's speed is looked after: its work, through the calls that its trainers and engines make.

An RL update of the default configuration (Qwen2.5-1.5B shapes, LoRA of rank 64, a DeBERTa-v3-large reward model) has four device
phases, and the cases follow them: generation (projections of a decode step, attention over fp8 or bf16 pages, sampling), scoring by
the reward model, log-probabilities without gradients, and the training micro-step (decoder layer, long-sequence attention at the 7B
model's heads, the fused log-probability head, the losses).  The step engine's families add windowed attention over pages and a
gated delta rule.

A case is a dict of plain values; ``kind`` names the builder.  Every builder makes its inputs from the seed alone.  ``exact`` gives
the same outputs by plain float64 torch.
"""
import math
import random

import numpy as np
import torch

from nanorlhf_b200 import _C, ops
from nanorlhf_b200.models.deberta_v3 import DebertaV3Config, DebertaV3ForSequenceClassification, build_bucket_lut
from nanorlhf_b200.models.lora import LoraConfig, get_peft_model
from nanorlhf_b200.models.qwen2 import Qwen2Config, Qwen2ForCausalLM
from nanorlhf_b200.ops import gemm, hybrid, native
from nanorlhf_b200.sampler.hybrid_sampler import StepPlan

DEV = "cuda"
VOCAB = 151936                      # Qwen2.5-1.5B
HIDDEN, FF, HEADS, KV_HEADS, HEAD = 1536, 8960, 12, 2, 128
RANK, ALPHA = 64, 16                # LoRA of the entry scripts
PAGE = 16


def listed():
    return [
        # one decoder layer of a training micro-step: four responses of unequal length with their prompts, forward and backward
        {"name": "policy_layer_train", "kind": "policy_layer", "train": True, "seqs": 4, "tokens": 6601},
        # the same layer in the log-probability pass over old and reference policy: no gradients, many sequences per chunk
        {"name": "policy_layer_logprob", "kind": "policy_layer", "train": False, "seqs": 22, "tokens": 32768},
        # attention of the 7B configuration over responses of up to 8000 tokens, forward and backward
        {"name": "attention_train_long", "kind": "attention", "heads": 28, "kv_heads": 4, "seqs": 2, "tokens": 12011},
        # the log-probability head of a micro-step: one row per response token against the whole vocabulary, forward and backward
        {"name": "logprob_head_train", "kind": "logprob_head", "rows": 6001},
        # one layer of the reward model over a batch of prompts with responses
        {"name": "reward_layer", "kind": "reward_layer", "seqs": 16, "tokens": 24571},
        # projections and norms of one layer in a decode step of a full batch
        {"name": "decode_projections", "kind": "projections", "rows": 1024},
        # attention of a decode step over fp8 pages (the sampler's default), full batch
        {"name": "decode_attention_fp8", "kind": "decode", "fp8": True, "seqs": 1024, "context": 1000},
        # the tail of a rollout: few sequences left, long contexts, bf16 pages, the key walk cut into parts
        {"name": "decode_attention_tail", "kind": "decode", "fp8": False, "seqs": 37, "context": 1500},
        # one token per sequence of a full batch: temperature 0.9, nucleus 0.95
        {"name": "sample_tokens", "kind": "sample", "rows": 1024},
        # advantages and both losses of a PPO micro-step, forward and backward: the smallest calls
        {"name": "ppo_losses", "kind": "losses", "seqs": 4, "response": 1500},
        # step engine, a prompt step: windowed attention over pages
        {"name": "paged_prompt_attention", "kind": "paged_attention", "heads": 16, "kv_heads": 4, "seqs": 16, "new": 2048, "old": 0,
         "window": 1024, "softcap": 0.0},
        # step engine, a prompt step: gated delta rule
        {"name": "delta_prompt", "kind": "delta", "heads": 16, "dim": 128, "seqs": 16, "new": 2048, "old": 0, "per_channel": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["policy_layer", "attention", "logprob_head", "reward_layer", "projections", "decode", "sample", "losses",
                       "paged_attention", "delta"])
    if kind == "policy_layer":
        train = rng.random() < 0.5
        seqs = rng.randint(1, 4) if train else rng.randint(1, 22)
        return {"kind": kind, "train": train, "seqs": seqs, "tokens": min(_log(rng, 200, 1650) * seqs + rng.randint(0, 99), 6600 if train else 32768)}
    if kind == "attention":
        heads, kv = rng.choice([(12, 2), (28, 4)])
        return {"kind": kind, "heads": heads, "kv_heads": kv, "seqs": (n := rng.randint(1, 6)), "tokens": min(_log(rng, 300, 11000), 8150 * n)}
    if kind == "logprob_head":
        return {"kind": kind, "rows": _log(rng, 100, 6000)}
    if kind == "reward_layer":
        seqs = rng.randint(2, 16)
        return {"kind": kind, "seqs": seqs, "tokens": _log(rng, 40, 1530) * seqs + rng.randint(0, 60)}
    if kind == "projections":
        return {"kind": kind, "rows": _log(rng, 8, 1024)}
    if kind == "decode":
        return {"kind": kind, "fp8": rng.random() < 0.5, "seqs": _log(rng, 4, 1000), "context": rng.randint(30, 1000)}
    if kind == "sample":
        return {"kind": kind, "rows": _log(rng, 4, 1020)}
    if kind == "losses":
        return {"kind": kind, "seqs": rng.randint(1, 32), "response": rng.randint(53, 1500)}
    if kind == "paged_attention":
        decode = rng.random() < 0.4
        return {"kind": kind, "heads": rng.choice([8, 16]), "kv_heads": rng.choice([2, 4]), "seqs": rng.randint(1, 16) if not decode else _log(rng, 4, 256),
                "new": 1 if decode else _log(rng, 70, 2000), "old": rng.randint(100, 2000) if decode else rng.choice([0, 0, 333, 1024]),
                "window": rng.choice([512, 1024, 100000]), "softcap": rng.choice([0.0, 0.0, 30.0])}
    decode = rng.random() < 0.4
    return {"kind": kind, "heads": rng.choice([8, 16]), "dim": rng.choice([64, 128]), "seqs": rng.randint(1, 16) if not decode else _log(rng, 4, 256),
            "new": 1 if decode else _log(rng, 70, 2000), "old": rng.randint(16, 2000) if decode else rng.choice([0, 0, 500]),
            "per_channel": rng.random() < 0.5}


# ---- helpers --------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * std).to(dtype)


def _lengths(total, n, seed):
    """``n`` unequal lengths that sum to ``total``."""
    r = random.Random(f"{total} {n} {seed}")
    w = [r.uniform(0.4, 1.0) for _ in range(n)]
    out = [max(1, int(total * x / sum(w))) for x in w]
    out[0] += total - sum(out)
    return out


def _cu(lens):
    return torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device=DEV)


def _positions(lens):
    return torch.cat([torch.arange(n, device=DEV) for n in lens])


def _causal_pairs(lens):
    return sum(n * (n + 1) / 2 for n in lens)


def _rms64(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _attention64(q, k, v, lens):
    """Causal grouped attention in float64, head by head; q [T, H, D], k / v [T, Hkv, D]."""
    group, scale, s0, out = q.shape[1] // k.shape[1], 1.0 / math.sqrt(q.shape[2]), 0, []
    for n in lens:
        heads = []
        mask = torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1)
        for h in range(q.shape[1]):
            s = (q[s0:s0 + n, h] @ k[s0:s0 + n, h // group].T * scale).masked_fill(mask, -math.inf)
            heads.append(torch.softmax(s, -1) @ v[s0:s0 + n, h // group])
        out.append(torch.stack(heads, 1))
        s0 += n
    return torch.cat(out)


# ---- decoder layer of the policy --------------------------------------------------------------------------------------------
_PROJ = [("self_attn.q_proj", HEADS * HEAD, HIDDEN), ("self_attn.k_proj", KV_HEADS * HEAD, HIDDEN), ("self_attn.v_proj", KV_HEADS * HEAD, HIDDEN),
         ("self_attn.o_proj", HIDDEN, HEADS * HEAD), ("mlp.gate_proj", FF, HIDDEN), ("mlp.up_proj", FF, HIDDEN), ("mlp.down_proj", HIDDEN, FF)]


def _policy_layer_inputs(case, seed):
    g = _gen(seed)
    w = {}
    for name, n, k in _PROJ:
        w[name] = _randn(g, n, k, std=0.02)
        w[name + ".A"] = _randn(g, RANK, k, std=1.0 / math.sqrt(3 * k))
        w[name + ".B"] = _randn(g, n, RANK, std=0.01)
        if name[-6:] in ("q_proj", "k_proj", "v_proj"):
            w[name + ".bias"] = _randn(g, n, std=0.1)
    for name in ("input_layernorm", "post_attention_layernorm"):
        w[name] = (1.0 + _randn(g, HIDDEN, std=0.1).float()).bfloat16()
    lens = _lengths(case["tokens"], case["seqs"], seed)
    return w, _randn(g, case["tokens"], HIDDEN), _randn(g, case["tokens"], HIDDEN, std=1e-2), lens


def _policy_layer_prepare(case, seed):
    w, x, gy, lens = _policy_layer_inputs(case, seed)
    cfg = Qwen2Config(vocab_size=256, num_hidden_layers=1)
    model = get_peft_model(Qwen2ForCausalLM.from_config(cfg, torch.bfloat16, DEV, seed=0), LoraConfig(r=RANK, lora_alpha=ALPHA))
    layer = model.base_model.model.layers[0]
    with torch.no_grad():
        for name, _, _ in _PROJ:
            m = layer.get_submodule(name)
            m.base_layer.weight.copy_(w[name])
            m.lora_A.weight.copy_(w[name + ".A"])
            m.lora_B.weight.copy_(w[name + ".B"])
            if name + ".bias" in w:
                m.base_layer.bias.copy_(w[name + ".bias"])
        layer.input_layernorm.weight.copy_(w["input_layernorm"])
        layer.post_attention_layernorm.weight.copy_(w["post_attention_layernorm"])
    cos, sin = ops.ref.rope_cos_sin(_positions(lens), HEAD, cfg.rope_theta)
    params = [layer.get_submodule(n).get_submodule(ab).weight for n, _, _ in _PROJ for ab in ("lora_A", "lora_B")]
    return {"layer": layer, "x": x.requires_grad_(case["train"]), "gy": gy, "cos": cos, "sin": sin, "cu": _cu(lens), "longest": max(lens),
            "params": params, "train": case["train"]}


def _policy_layer_run(s):
    if not s["train"]:
        with torch.no_grad():
            return s["layer"](s["x"], s["cos"], s["sin"], s["cu"], s["longest"])
    y = s["layer"](s["x"], s["cos"], s["sin"], s["cu"], s["longest"])
    return [y.detach()] + list(torch.autograd.grad(y, [s["x"]] + s["params"], s["gy"]))


def _policy_layer_exact(case, seed):
    w, x, gy, lens = _policy_layer_inputs(case, seed)
    w = {k: v.double() for k, v in w.items()}
    x = x.double().requires_grad_(case["train"])
    ab = [w[n + "." + c].requires_grad_(case["train"]) for n, _, _ in _PROJ for c in "AB"]
    inv = 1.0 / (1e6 ** (torch.arange(0, HEAD, 2, device=DEV, dtype=torch.float64) / HEAD))
    ang = _positions(lens).double()[:, None] * inv
    cos, sin = torch.cat([ang, ang], 1).cos()[:, None], torch.cat([ang, ang], 1).sin()[:, None]

    def lin(h, n):
        y = h @ w[n].T + (h @ w[n + ".A"].T) @ w[n + ".B"].T * (ALPHA / RANK)
        return y + w[n + ".bias"] if n + ".bias" in w else y

    def rope(t):
        a, b = t.chunk(2, -1)
        return t * cos + torch.cat([-b, a], -1) * sin

    with torch.set_grad_enabled(case["train"]):
        T, h = case["tokens"], _rms64(x, w["input_layernorm"], 1e-6)
        q, k, v = (lin(h, "self_attn." + n).view(T, -1, HEAD) for n in ("q_proj", "k_proj", "v_proj"))
        x1 = x + lin(_attention64(rope(q), rope(k), v, lens).reshape(T, -1), "self_attn.o_proj")
        h = _rms64(x1, w["post_attention_layernorm"], 1e-6)
        y = x1 + lin(torch.nn.functional.silu(lin(h, "mlp.gate_proj")) * lin(h, "mlp.up_proj"), "mlp.down_proj")
    if not case["train"]:
        return y
    return [y.detach()] + list(torch.autograd.grad(y, [x] + ab, gy.double()))


def _policy_layer_work(case):
    T, lens = case["tokens"], _lengths(case["tokens"], case["seqs"], 0)
    weights = sum(n * k for _, n, k in _PROJ)
    lora = sum((n + k) * RANK for _, n, k in _PROJ)
    lin = 2.0 * T * weights * (2 if case["train"] else 1) + 2.0 * T * lora * (3 if case["train"] else 1)      # the base weights are frozen
    att = 4.0 * HEADS * HEAD * _causal_pairs(lens) * (3.5 if case["train"] else 1)
    return {"bytes": 2.0 * (weights + lora * (2 if case["train"] else 1)) + 2.0 * T * HIDDEN * (4 if case["train"] else 2), "flops": lin + att}


# ---- training attention -----------------------------------------------------------------------------------------------------
def _attention_inputs(case, seed):
    g, T = _gen(seed), case["tokens"]
    q, k, v = _randn(g, T, case["heads"], HEAD), _randn(g, T, case["kv_heads"], HEAD), _randn(g, T, case["kv_heads"], HEAD)
    return q, k, v, _randn(g, T, case["heads"], HEAD), _lengths(T, case["seqs"], seed)


def _attention_prepare(case, seed):
    q, k, v, do, lens = _attention_inputs(case, seed)
    return {"qkv": [t.requires_grad_(True) for t in (q, k, v)], "do": do, "cu": _cu(lens), "longest": max(lens)}


def _attention_run(s):
    o = ops.attention_varlen(*s["qkv"], s["cu"], s["longest"])
    return [o.detach()] + list(torch.autograd.grad(o, s["qkv"], s["do"]))


def _attention_exact(case, seed):
    """Forward and backward head by head (the score matrix of a long sequence is half a gigabyte)."""
    q, k, v, do, lens = _attention_inputs(case, seed)
    group, scale = case["heads"] // case["kv_heads"], 1.0 / math.sqrt(HEAD)
    o, dq, dk, dv = (torch.zeros(t.shape, dtype=torch.float64, device=DEV) for t in (q, q, k, v))
    s0 = 0
    for n in lens:
        r, mask = slice(s0, s0 + n), torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1)
        for h in range(case["heads"]):
            qh, kh, vh, gh = q[r, h].double(), k[r, h // group].double(), v[r, h // group].double(), do[r, h].double()
            p = torch.softmax((qh @ kh.T * scale).masked_fill_(mask, -math.inf), -1)
            o[r, h] = p @ vh
            ds = p * (gh @ vh.T - (gh * o[r, h]).sum(-1, keepdim=True)) * scale
            dq[r, h] = ds @ kh
            dk[r, h // group] += ds.T @ qh
            dv[r, h // group] += p.T @ gh
        s0 += n
    return [o, dq, dk, dv]


def _attention_work(case):
    T, H, Hkv = case["tokens"], case["heads"], case["kv_heads"]
    pairs = _causal_pairs(_lengths(T, case["seqs"], 0))
    return {"bytes": 2.0 * T * HEAD * (4 * H + 4 * Hkv), "flops": 14.0 * H * HEAD * pairs}      # 2 products forward, 5 backward


# ---- log-probability head ---------------------------------------------------------------------------------------------------
def _head_inputs(case, seed):
    g, R = _gen(seed), case["rows"]
    return (_randn(g, R, HIDDEN), _randn(g, VOCAB, HIDDEN, std=0.05), torch.randint(0, VOCAB, (R,), generator=g, device=DEV),
            torch.randn(R, generator=g, device=DEV) / R)


def _head_prepare(case, seed):
    h, w, t, gl = _head_inputs(case, seed)
    return {"h": h.requires_grad_(True), "w": w.requires_grad_(True), "t": t, "g": gl}


def _head_run(s):
    logp, ent = ops.lmhead_logprob(s["h"], s["w"], s["t"], 0.9)
    return [logp.detach(), ent] + list(torch.autograd.grad(logp, [s["h"], s["w"]], s["g"]))


def _head_exact(case, seed):
    h, w, t, gl = _head_inputs(case, seed)
    h, w, gl = h.double(), w.double(), gl.double()
    logp, ent = torch.empty_like(gl), torch.empty_like(gl)
    dh, dw = torch.empty_like(h), torch.zeros_like(w)
    for a in range(0, len(t), 1024):
        r = slice(a, a + 1024)
        lp = torch.log_softmax(h[r] @ w.T / 0.9, -1)
        p = lp.exp()
        logp[r] = lp.gather(1, t[r, None])[:, 0]
        ent[r] = -(p * lp).sum(-1)
        dz = p.mul_(-gl[r, None] / 0.9)
        dz.scatter_add_(1, t[r, None], gl[r, None] / 0.9)
        dh[r] = dz @ w
        dw += dz.T @ h[r]
    return [logp, ent, dh, dw]


def _head_work(case):
    R = case["rows"]
    return {"bytes": 2.0 * (2 * R * HIDDEN + 2 * VOCAB * HIDDEN) + 16.0 * R, "flops": 6.0 * R * VOCAB * HIDDEN}


# ---- reward model layer -----------------------------------------------------------------------------------------------------
_RM = DebertaV3Config.large()
_RM_LINEAR = ["attention.self.query_proj", "attention.self.key_proj", "attention.self.value_proj", "attention.output.dense",
              "intermediate.dense", "output.dense"]


def _reward_inputs(case, seed):
    g, W = _gen(seed), _RM.hidden_size
    w = {}
    for n in _RM_LINEAR:
        rows, cols = (_RM.intermediate_size, W) if n.startswith("inter") else (W, _RM.intermediate_size) if n == "output.dense" else (W, W)
        w[n + ".weight"], w[n + ".bias"] = _randn(g, rows, cols, std=0.04), _randn(g, rows, std=0.1)
    for n in ("attention.output.LayerNorm", "output.LayerNorm"):
        w[n + ".weight"], w[n + ".bias"] = (1.0 + _randn(g, W, std=0.1).float()).bfloat16(), _randn(g, W, std=0.1)
    lens = _lengths(case["tokens"], case["seqs"], seed)
    return w, _randn(g, case["tokens"], W), _randn(g, 2 * _RM.position_buckets, W, std=0.5), lens


def _reward_prepare(case, seed):
    w, x, rel, lens = _reward_inputs(case, seed)
    cfg = DebertaV3Config(vocab_size=64, num_hidden_layers=1)
    layer = DebertaV3ForSequenceClassification.from_config(cfg, torch.bfloat16, DEV, seed=0).deberta.encoder.layer[0]
    with torch.no_grad():
        for n, p in layer.named_parameters():
            p.copy_(w[n])
    lut = build_bucket_lut(max(lens), cfg.position_buckets, cfg.max_position_embeddings, cfg.position_buckets, DEV)
    return {"layer": layer, "x": x, "rel": rel, "cu": _cu(lens), "longest": max(lens), "lut": lut}


def _reward_run(s):
    layer, x = s["layer"], s["x"]
    with torch.no_grad():
        a = layer.attention.self.forward_packed(x, s["cu"], s["longest"], s["lut"], s["rel"])
        a = layer.attention.output(a, x)
        return layer.output(layer.intermediate(a), a)


def _reward_exact(case, seed):
    w, x, rel, lens = _reward_inputs(case, seed)
    w, x, rel = {k: v.double() for k, v in w.items()}, x.double(), rel.double()
    H, span = _RM.num_attention_heads, _RM.position_buckets
    F = torch.nn.functional

    def lin(t, n):
        return t @ w[n + ".weight"].T + w[n + ".bias"]

    def heads(t):
        return t.view(-1, H, 64).transpose(0, 1)

    def bucket(d):
        mid, top = span // 2, _RM.max_position_embeddings
        far = torch.ceil(torch.log(d.abs().clamp(min=mid).float() / mid) / math.log((top - 1) / mid) * (mid - 1)) + mid
        return torch.where(d.abs() <= mid, d, (far * d.sign()).long())

    q, k, v = (heads(lin(x, "attention.self." + n)) for n in ("query_proj", "key_proj", "value_proj"))
    pk, pq = heads(lin(rel, "attention.self.key_proj")), heads(lin(rel, "attention.self.query_proj"))
    out, s0 = [], 0
    for n in lens:
        i = torch.arange(n, device=DEV)
        idx = (bucket(i[:, None] - i[None, :]) + span).clamp(0, 2 * span - 1)
        rows = []
        for h in range(H):
            qh, kh, vh = q[h, s0:s0 + n], k[h, s0:s0 + n], v[h, s0:s0 + n]
            s = qh @ kh.T + (qh @ pk[h].T).gather(1, idx) + (kh @ pq[h].T).gather(1, idx.T).T
            rows.append(torch.softmax(s / math.sqrt(192.0), -1) @ vh)
        out.append(torch.stack(rows, 1).reshape(n, -1))
        s0 += n
    ln = lambda t, n: F.layer_norm(t, (_RM.hidden_size,), w[n + ".weight"], w[n + ".bias"], _RM.layer_norm_eps)  # noqa: E731
    a = ln(lin(torch.cat(out), "attention.output.dense") + x, "attention.output.LayerNorm")
    return ln(lin(F.gelu(lin(a, "intermediate.dense")), "output.dense") + a, "output.LayerNorm")


def _reward_work(case):
    T, W = case["tokens"], _RM.hidden_size
    weights = 4 * W * W + 2 * W * _RM.intermediate_size
    lens = _lengths(T, case["seqs"], 0)
    tables = 4.0 * T * W * 2 * _RM.position_buckets            # queries and keys against the 512 relative positions
    return {"bytes": 2.0 * weights + 4.0 * T * W, "flops": 2.0 * T * weights + tables + 4.0 * W * sum(n * n for n in lens)}


# ---- projections of a decode step -------------------------------------------------------------------------------------------
def _proj_inputs(case, seed):
    g, S = _gen(seed), case["rows"]
    return {"x": _randn(g, S, HIDDEN), "res": _randn(g, S, HIDDEN), "att": _randn(g, S, HEADS * HEAD),
            "ln1": (1.0 + _randn(g, HIDDEN, std=0.1).float()).bfloat16(), "ln2": (1.0 + _randn(g, HIDDEN, std=0.1).float()).bfloat16(),
            "wqkv": _randn(g, (HEADS + 2 * KV_HEADS) * HEAD, HIDDEN, std=0.02), "bqkv": _randn(g, (HEADS + 2 * KV_HEADS) * HEAD, std=0.1),
            "wo": _randn(g, HIDDEN, HEADS * HEAD, std=0.02), "wg": _randn(g, FF, HIDDEN, std=0.02), "wu": _randn(g, FF, HIDDEN, std=0.02),
            "wdown": _randn(g, HIDDEN, FF, std=0.02)}


def _proj_prepare(case, seed):
    s = _proj_inputs(case, seed)
    s["wgu"] = torch.stack([s.pop("wg").view(FF // 32, 32, HIDDEN), s.pop("wu").view(FF // 32, 32, HIDDEN)], 1).reshape(2 * FF, HIDDEN)
    return s


def _proj_run(s):
    """The linear side of a layer as the sampler runs it; ``att`` stands for the attention's result."""
    with torch.no_grad():
        h, res = native.add_rmsnorm(s["x"], s["res"], s["ln1"], 1e-6)
        qkv = gemm.gemm(h, s["wqkv"], bias=s["bqkv"])
        o = gemm.gemm(s["att"], s["wo"])
        h, res = native.add_rmsnorm(o, res, s["ln2"], 1e-6)
        act = native.ext().gemm_tc_swiglu(h, s["wgu"], None)
        return qkv, gemm.gemm(act, s["wdown"]), res


def _proj_exact(case, seed):
    s = {k: v.double() for k, v in _proj_inputs(case, seed).items()}
    res = s["x"] + s["res"]
    qkv = _rms64(res, s["ln1"], 1e-6) @ s["wqkv"].T + s["bqkv"]
    res = res + s["att"] @ s["wo"].T
    h = _rms64(res, s["ln2"], 1e-6)
    return qkv, (torch.nn.functional.silu(h @ s["wg"].T) * (h @ s["wu"].T)) @ s["wdown"].T, res


def _proj_work(case):
    S, n = case["rows"], sum(a * b for _, a, b in _PROJ)
    return {"bytes": 2.0 * n + 2.0 * S * (5 * HIDDEN + (HEADS + 2 * KV_HEADS) * HEAD), "flops": 2.0 * S * n}


# ---- decode attention -------------------------------------------------------------------------------------------------------
def _decode_inputs(case, seed):
    g, S = _gen(seed), case["seqs"]
    r = random.Random(f"{S} {seed}")
    lens = [max(1, int(case["context"] * r.uniform(0.5, 1.5))) for _ in range(S)]
    width = (max(lens) + PAGE - 1) // PAGE
    used = [(n + PAGE - 1) // PAGE for n in lens]
    order = torch.randperm(sum(used), generator=g, device=DEV).int()         # pages of a sequence lie anywhere in the pool
    table, o = torch.zeros(S, width, dtype=torch.int32, device=DEV), 0
    for i, n in enumerate(used):
        table[i, :n] = order[o:o + n]
        o += n
    shape = (sum(used), KV_HEADS, PAGE, HEAD)
    k, v = _randn(g, *shape), _randn(g, *shape)
    s = {"q": _randn(g, S, HEADS, HEAD), "table": table, "lens": torch.tensor(lens, dtype=torch.int32, device=DEV)}
    if case["fp8"]:                                                          # e4m3 pages, values transposed in the page, a scale per token
        k, v = k * 100, (v * 100).transpose(2, 3).contiguous()
        s["ks"], s["vs"] = (torch.rand(shape[:3], generator=g, device=DEV) * 0.01 + 0.005 for _ in range(2))
        k, v = k.clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8), v.clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    s["k"], s["v"] = k, v
    return s


def _decode_prepare(case, seed):
    s = _decode_inputs(case, seed)
    rows = case["seqs"] * KV_HEADS                       # the sampler's rule for the number of parts of the key walk
    s["splits"] = 1 if rows >= 296 else int(min(8, max(1, math.ceil(296 / max(1, rows)))))
    return s


def _decode_run(s):
    if "ks" in s:
        return native.ext().paged_decode_fp8(s["q"], s["k"], s["v"], s["ks"], s["vs"], s["table"], s["lens"], 1.0 / math.sqrt(HEAD), s["splits"])
    return native.paged_decode(s["q"], s["k"], s["v"], s["table"], s["lens"], 1.0 / math.sqrt(HEAD), s["splits"])


def _decode_exact(case, seed):
    s = _decode_inputs(case, seed)
    k, v = s["k"], s["v"]
    if case["fp8"]:
        k = k.view(torch.float8_e4m3fn).float() * s["ks"][..., None]
        v = v.view(torch.float8_e4m3fn).float().transpose(2, 3) * s["vs"][..., None]
    out = []
    for i, n in enumerate(s["lens"].tolist()):
        pages = s["table"][i, :(n + PAGE - 1) // PAGE].long()
        kk, vv = (t[pages].transpose(0, 1).reshape(KV_HEADS, -1, HEAD)[:, :n].double() for t in (k, v))
        q = s["q"][i].double().view(KV_HEADS, HEADS // KV_HEADS, HEAD)
        out.append((torch.softmax(q @ kk.transpose(1, 2) / math.sqrt(HEAD), -1) @ vv).reshape(HEADS, HEAD))
    return torch.stack(out)


def _decode_work(case):
    tokens, per = case["seqs"] * case["context"], KV_HEADS * (2 * HEAD + 8 if case["fp8"] else 4 * HEAD)
    return {"bytes": float(tokens * per + case["seqs"] * HEADS * HEAD * 4), "flops": 4.0 * tokens * HEADS * HEAD}


# ---- sampling ---------------------------------------------------------------------------------------------------------------
def _sample_prepare(case, seed):
    g, R = _gen(seed), case["rows"]
    sharp = torch.rand(R, 1, generator=g, device=DEV) * 3 + 1                # from nearly flat rows to confident ones
    return {"logits": (torch.randn(R, VOCAB, generator=g, device=DEV) * sharp).bfloat16(), "ids": torch.arange(R, dtype=torch.int32, device=DEV),
            "steps": torch.randint(0, 1500, (R,), generator=g, device=DEV).int(), "seed": int(seed)}


def _sample_run(s):
    return native.sample(s["logits"], 0.9, 0.95, s["seed"], 0, s["ids"], s["steps"])


def _sample_work(case):
    return {"bytes": case["rows"] * (2.0 * VOCAB + 12), "flops": 4.0 * case["rows"] * VOCAB}


# ---- losses -----------------------------------------------------------------------------------------------------------------
GAMMA, LAM, CLIP, KL = 1.0, 0.95, 0.2, 0.01


def _loss_inputs(case, seed):
    g, B, T = _gen(seed), case["seqs"], case["response"]
    f = lambda std: torch.randn(B, T, generator=g, device=DEV) * std  # noqa: E731
    lens = torch.randint(T // 2, T + 1, (B, 1), generator=g, device=DEV)
    mask = torch.arange(T, device=DEV)[None] < lens
    old = -f(1.0).abs()
    return {"new": old + f(0.15), "old": old, "ref": old + f(0.1), "rewards": f(0.3) * mask, "values": f(0.5), "vpred": f(0.5), "mask": mask}


def _loss_prepare(case, seed):
    s = _loss_inputs(case, seed)
    s["new"].requires_grad_(True)
    s["vpred"].requires_grad_(True)
    return s


def _loss_run(s):
    adv, ret = ops.gae(s["rewards"], s["values"], GAMMA, LAM)
    loss, _stats = ops.policy_loss_token(s["new"], s["old"], adv, s["mask"], CLIP, s["ref"], KL)
    vloss, clipfrac = ops.value_loss(s["vpred"], s["values"], ret, s["mask"], CLIP)
    return [adv, ret, loss.detach(), vloss.detach(), clipfrac] + list(torch.autograd.grad(loss + 0.1 * vloss, [s["new"], s["vpred"]]))


def _loss_exact(case, seed):
    s = _loss_inputs(case, seed)
    m = s.pop("mask").double()
    s = {k: v.double() for k, v in s.items()}
    nxt = torch.cat([s["values"][:, 1:], torch.zeros_like(s["values"][:, :1])], 1)
    delta, adv, last = s["rewards"] + GAMMA * nxt - s["values"], torch.empty_like(nxt), 0.0
    for t in range(nxt.shape[1] - 1, -1, -1):
        last = delta[:, t] + GAMMA * LAM * last
        adv[:, t] = last
    ret = adv + s["values"]
    new, vp = s["new"].requires_grad_(True), s["vpred"].requires_grad_(True)
    ratio, k = torch.exp(new - s["old"]), new - s["ref"]
    per = torch.maximum(-adv * ratio, -adv * ratio.clamp(1 - CLIP, 1 + CLIP)) + KL * (torch.exp(-k) + k - 1)
    loss = (per * m).sum() / m.sum()
    vc = torch.maximum(torch.minimum(vp, s["values"] + CLIP), s["values"] - CLIP)
    l1, l2 = (vp - ret) ** 2, (vc - ret) ** 2
    vloss = 0.5 * (torch.maximum(l1, l2) * m).sum() / m.sum()
    clipfrac = ((l2 > l1).double() * m).sum() / m.sum()
    return [adv, ret, loss.detach(), vloss.detach(), clipfrac] + list(torch.autograd.grad(loss + 0.1 * vloss, [new, vp]))


def _loss_work(case):
    n = case["seqs"] * case["response"]
    return {"bytes": n * (6 * 4.0 + 1 + 4 * 4.0), "flops": 40.0 * n}


# ---- step engine ------------------------------------------------------------------------------------------------------------
def _plan(case):
    """The packed plan of a step in which every sequence has ``new`` tokens behind ``old`` earlier ones; pages in the pool."""
    B, n, old = case["seqs"], case["new"], case["old"]
    pages = (old + n + PAGE - 1) // PAGE * B + 8
    sched = _C.StepScheduler(pages, PAGE, B)
    ids = [sched.open() for _ in range(B)]
    if old:
        sched.plan(ids, [old] * B)
    data, E, T, width = sched.plan(ids, [n] * B)
    return StepPlan(torch.from_numpy(data).to(DEV), E, T, width), pages


def _paged_inputs(case, seed):
    plan, pages = _plan(case)
    g, H, Hkv = _gen(seed), case["heads"], case["kv_heads"]
    return plan, _randn(g, plan.T, H * HEAD, dtype=torch.float32), _randn(g, pages, Hkv, PAGE, HEAD), _randn(g, pages, Hkv, PAGE, HEAD)


def _paged_prepare(case, seed):
    plan, q, k, v = _paged_inputs(case, seed)
    return {"plan": plan, "q": q, "k": k, "v": v, "window": case["window"], "softcap": case["softcap"],
            "out": torch.empty(plan.T, case["heads"] * HEAD, dtype=torch.bfloat16, device=DEV)}


def _paged_run(s):
    hybrid.window_attention(s["q"], s["k"], s["v"], s["plan"], s["window"], HEAD ** -0.5, 1.0, s["out"], softcap=s["softcap"])
    return s["out"]


def _paged_exact(case, seed):
    plan, q, k, v = _paged_inputs(case, seed)
    H, Hkv, n, old = case["heads"], case["kv_heads"], case["new"], case["old"]
    total, out = old + n, torch.empty(plan.T, H, HEAD, dtype=torch.float64, device=DEV)
    qp, kp = torch.arange(old, total, device=DEV)[:, None], torch.arange(total, device=DEV)[None]
    hidden = (kp > qp) | (kp <= qp - case["window"])
    for e in range(case["seqs"]):
        pages = plan.block_table[e, :(total + PAGE - 1) // PAGE].long()
        kk, vv = (t[pages].transpose(0, 1).reshape(Hkv, -1, HEAD)[:, :total].double() for t in (k, v))
        for h in range(H):
            r = slice(e * n, (e + 1) * n)
            s = q[r, h * HEAD:(h + 1) * HEAD].double() @ kk[h * Hkv // H].T * HEAD ** -0.5
            if case["softcap"]:
                s = case["softcap"] * torch.tanh(s / case["softcap"])
            out[r, h] = torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ vv[h * Hkv // H]
    return out.reshape(plan.T, -1)


def _paged_work(case):
    B, n, old, H, Hkv = (case[x] for x in ("seqs", "new", "old", "heads", "kv_heads"))
    pairs = B * sum(min(p + 1, case["window"]) for p in range(old, old + n))
    keys = B * min(old + n, case["window"] + n - 1)
    return {"bytes": B * n * H * HEAD * 6.0 + keys * Hkv * HEAD * 4.0, "flops": 4.0 * pairs * H * HEAD}


def _delta_inputs(case, seed):
    plan, _ = _plan(case)
    g, T, H, D = _gen(seed), plan.T, case["heads"], case["dim"]
    f = lambda *shape: torch.randn(*shape, generator=g, device=DEV)  # noqa: E731
    q, k = (torch.nn.functional.normalize(f(T, H, D), dim=-1) for _ in range(2))
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), f(T, H * D)], 1).contiguous()
    beta = torch.sigmoid(f(T, H))
    decay = torch.exp(-torch.nn.functional.softplus(f(T, H * D if case["per_channel"] else H) - 3))
    state = f(case["seqs"], H, D, D) * 0.3
    return plan, qkv, beta, decay, state


def _delta_prepare(case, seed):
    plan, qkv, beta, decay, state = _delta_inputs(case, seed)
    return {"plan": plan, "qkv": qkv, "beta": beta, "decay": decay, "state": state, "heads": case["heads"], "dim": case["dim"],
            "per_channel": case["per_channel"], "o": torch.empty(plan.T, case["heads"] * case["dim"], device=DEV)}


def _delta_run(s):
    c = s["heads"] * s["dim"]
    hybrid.delta_scan(s["qkv"], c, 2 * c, s["beta"], s["decay"], s["state"], s["o"], s["plan"], s["heads"], s["per_channel"])
    return s["o"], s["state"]


def _delta_exact(case, seed):
    plan, qkv, beta, decay, state = _delta_inputs(case, seed)
    B, n, H, D = case["seqs"], case["new"], case["heads"], case["dim"]
    q, k, v = (t.double().view(B, n, H, D) for t in qkv.chunk(3, 1))
    beta, decay = beta.double().view(B, n, H, 1), decay.double().view(B, n, H, -1, 1)
    slots = plan.state_slot.long()
    S = state[slots].double() if case["old"] else torch.zeros(B, H, D, D, dtype=torch.float64, device=DEV)
    o = torch.empty(B, n, H, D, dtype=torch.float64, device=DEV)
    for t in range(n):
        S = S * decay[:, t]
        kt = k[:, t, :, :, None]
        u = beta[:, t] * (v[:, t] - (S * kt).sum(-2))
        S = S + kt * u[:, :, None]
        o[:, t] = (S * q[:, t, :, :, None]).sum(-2)
    out = state.double()
    out[slots] = S
    return o.reshape(B * n, -1), out


def _delta_work(case):
    B, n, H, D = case["seqs"], case["new"], case["heads"], case["dim"]
    per = 4 * H * D + H + (H * D if case["per_channel"] else H)
    return {"bytes": B * n * per * 4.0 + (2 if case["old"] else 1) * B * H * D * D * 4.0, "flops": 8.0 * B * n * H * D * D}


# ---- the five entry points --------------------------------------------------------------------------------------------------
# Tolerances: relative error over the result's norm, about four times what two correct implementations at the same precision differ by.
# bf16 operands with float32 sums give 2e-3 to 4e-3 a product, and a layer is a chain of them; float32 work differs in the order of sums.
_KINDS = {
    "policy_layer": (_policy_layer_prepare, _policy_layer_run, _policy_layer_exact, _policy_layer_work, {"rel": 2.5e-2}),
    "attention": (_attention_prepare, _attention_run, _attention_exact, _attention_work, {"rel": 1.5e-2}),
    "logprob_head": (_head_prepare, _head_run, _head_exact, _head_work, {"rel": 1.2e-2}),
    "reward_layer": (_reward_prepare, _reward_run, _reward_exact, _reward_work, {"rel": 1.5e-2}),
    "projections": (_proj_prepare, _proj_run, _proj_exact, _proj_work, {"rel": 1.2e-2}),
    "decode": (_decode_prepare, _decode_run, _decode_exact, _decode_work, {"rel": 1e-2}),
    "sample": (_sample_prepare, _sample_run, lambda case, seed: None, _sample_work, {"rel": 0.0, "max": 0.0, "differ": 5e-3}),
    "losses": (_loss_prepare, _loss_run, _loss_exact, _loss_work, {"rel": 2e-5, "max": 2e-4}),
    "paged_attention": (_paged_prepare, _paged_run, _paged_exact, _paged_work, {"rel": 1.2e-2}),
    "delta": (_delta_prepare, _delta_run, _delta_exact, _delta_work, {"rel": 1e-5, "max": 1e-3}),
}


def prepare(case, seed):
    return dict(_KINDS[case["kind"]][0](case, seed), kind=case["kind"])


def run(state):
    return _KINDS[state["kind"]][1](state)


def exact(case, seed):
    return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


def tolerance(case):
    return _KINDS[case["kind"]][4]
