"""Linear layers of the training / log-prob / reward paths on the general tcgen05 GEMM (csrc/gemm_tc.cu).

What the reference runs here is cuBLAS behind ``nn.Linear`` plus peft's LoRA wrapper -- per projection and direction a base
GEMM, two adapter GEMMs and an add over the ``[tokens, out]`` result (GRPO/grpo.py:228-243; call sites
GRPO/grpo_trainer.py:543-556,652-660).  Here every contraction of the decoder is one launch of the same
sm_100a kernel, with the operand "major-ness" chosen so that no transposed copy is ever made:

=================  =========================================  =====================================================
 product            operands as stored                         kernel form
=================  =========================================  =====================================================
 y  = x W^T (+b)    x [T,K], W [N,K]                           K-major x K-major
 dx = dy W          dy [T,N], W [N,K] = [contraction, out]     K-major x MN-major
 dW = dy^T x        dy [T,N], x [T,K]  (tokens = contraction)  MN-major x MN-major
 LoRA forward       t = s x A^T;  y = [x | t] [W | B]^T        dual-source K: ONE GEMM with K + r columns
 LoRA dgrad         t' = s dy B;  dx = [dy | t'] [W ; A]       dual-source K, MN-major B operands
 LoRA wgrad         dA = t'^T x,  dB = dy^T t                  MN-major x MN-major (rank-r outputs)
=================  =========================================  =====================================================

Projections of one input share a launch (``_projections``), so do the products whose sum is that input's gradient (``sum_gemms``) and the narrow
gradients of a group's factors (``_adapter_grads``).

Tensors whose shape the kernel cannot address (inner extents not multiples of 8, mis-aligned rows) and non-bf16 /
non-CUDA tensors take the PyTorch path; a bf16 CUDA tensor of a supported shape never falls back silently.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from . import native as _native_mod


def _ok2d(t: torch.Tensor) -> bool:
    return (t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0
            and t.shape[0] > 0 and t.shape[1] % 8 == 0)


def supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    from . import use_native
    return (use_native(x) and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and w.dim() == 2
            and w.shape[0] % 8 == 0 and w.shape[1] % 8 == 0 and w.is_contiguous() and x.shape[-1] == w.shape[1])


def _rows(x: torch.Tensor) -> torch.Tensor:
    x2 = x.reshape(-1, x.shape[-1])
    return x2 if _ok2d(x2) else x2.contiguous()


def gemm(a, b, a_mn=False, b_mn=False, a2=None, b2=None, bias=None, act=0, alpha=1.0, out=None, out_f32=None,
         accumulate=False, cg=0, block_n=0, split_k=-1, residual=None):
    """Thin wrapper over ``_C.gemm_tc`` (see csrc/bindings.cpp) that counts the launch."""
    _native_mod._count()
    return _native_mod.ext().gemm_tc(a, b, a_mn, b_mn, a2, b2, bias, act, alpha, out, out_f32, accumulate, cg, block_n,
                                     split_k, residual)


class _LinearFn(torch.autograd.Function):
    """y = x W^T + b; forward, dgrad and wgrad on the tcgen05 kernel, no transposed copies."""

    @staticmethod
    def forward(ctx, x, w, b, act):
        x2 = _rows(x)
        y = gemm(x2, w, bias=b, act=act)
        ctx.save_for_backward(x2, w)
        ctx.has_bias = b is not None
        ctx.xshape = x.shape
        if act != 0:
            ctx.mark_non_differentiable(y)           # the fused activation is inference-only (reward model)
        return y.view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, gy):
        x2, w = ctx.saved_tensors
        g2 = _rows(gy)
        gx = gw = gb = None
        if ctx.needs_input_grad[0]:
            gx = gemm(g2, w, b_mn=True).view(ctx.xshape)
        if ctx.needs_input_grad[1]:
            gw = gemm(g2, x2, a_mn=True, b_mn=True)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            gb = g2.float().sum(0).to(g2.dtype)
        return gx, gw, gb, None


def linears(x, ws, bs):
    """``[F.linear(x, w, b) ...]`` of one input without autograd; None where the native GEMMs do not apply or add up ranges of a contraction."""
    if x.numel() == 0 or not all(supported(x, w) for w in ws):
        return None
    x2 = _rows(x)
    pick, dev = _native_mod.ext().gemm_tc_auto_splits, x2.get_device()
    if any(pick(x2.shape[0], *shape, dev) > 1 for shape in {w.shape for w in ws}):
        return None
    return [y.view(*x.shape[:-1], y.shape[-1]) for y in _projections(x2, ws, bs)]


def linear(x, w, b=None, act: int = 0):
    """``F.linear`` on the native GEMM (``act=1``: exact GELU fused into the epilogue, no-grad use only)."""
    if supported(x, w):
        return _LinearFn.apply(x, w, b, act)
    y = F.linear(x, w, b)
    return F.gelu(y) if act == 1 else y


class _LoraLinearFn(torch.autograd.Function):
    """y = x W^T + b + s (x A^T) B^T with a frozen W: the adapter rides in the base GEMM as extra contraction columns."""

    @staticmethod
    def forward(ctx, x, w, bias, a, b, scaling):
        x2 = _rows(x)
        t = gemm(x2, a, alpha=scaling)                                   # [T, r] = s x A^T
        y = gemm(x2, w, a2=t, b2=b, bias=bias)                           # [x | t] [W | B]^T
        ctx.save_for_backward(x2, w, a, b, t)
        ctx.scaling = scaling
        ctx.xshape = x.shape
        return y.view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, gy):
        x2, w, a, b, t = ctx.saved_tensors
        s = ctx.scaling
        g2 = _rows(gy)
        tp = gemm(g2, b, b_mn=True, alpha=s)                             # [T, r] = s dy B
        gx = ga = gb = None
        if ctx.needs_input_grad[0]:
            gx = gemm(g2, w, b_mn=True, a2=tp, b2=a).view(ctx.xshape)    # [dy | t'] [W ; A]
        # dA = t'^T x [r, K] (s is inside t'), dB = dy^T t [N, r] (s is inside t)
        gbs, gas = _adapter_grads([(g2, t)] if ctx.needs_input_grad[4] else [], [(tp, x2)] if ctx.needs_input_grad[3] else [], a.shape[0])
        ga, gb = gas[0] if gas else None, gbs[0] if gbs else None
        return gx, None, None, ga, gb, None


def lora_supported(x, w, a, b) -> bool:
    return (supported(x, w) and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and a.is_contiguous()
            and b.is_contiguous() and a.shape[0] % 8 == 0 and a.shape[0] == b.shape[1])


def lora_linear(x, w, bias, a, b, scaling: float):
    return _LoraLinearFn.apply(x, w, bias, a, b, float(scaling))


def sum_gemms(a, b):
    """``sum_i a[i] b[i]`` for the gradient of an input that several projections share: one launch with one float accumulator where none of the
    products would be cut into ranges of its contraction, else product by product, added in bf16."""
    pick, rows, cols, dev = _native_mod.ext().gemm_tc_auto_splits, a[0].shape[0], b[0].shape[1], a[0].get_device()
    if len(a) <= 4 and all(pick(rows, cols, k, dev) == 1 for k in {x.shape[1] for x in a}):
        _native_mod._count()
        return _native_mod.ext().gemm_tc_sum(a, b)
    out = gemm(a[0], b[0], b_mn=True, a2=a[-1], b2=b[-1])
    for x, y in zip(a[1:-1], b[1:-1]):
        out = out + gemm(x, y, b_mn=True)
    return out


def _narrow(r: int) -> bool:
    """Whether an adapter's products may share launches, in tiles 64 wide.  Wider factors fill wider tiles by themselves: rank 32 at 6601 tokens of a
    1536 / 8960 wide MLP 88 -> 66 us in one launch, rank 64 87 -> 69, rank 128 95 -> 107, rank 256 121 -> 187."""
    return r <= 64


def _multi(a, b, out, flip, alpha: float, a_mn: bool):
    """``out_i = alpha a_i b_i`` (``a_mn``: ``alpha a_i^T b_i``, the transpose of it where ``flip`` says so), up to six in a launch where that is faster than a GEMM each."""
    ext = _native_mod.ext()
    for i in range(0, len(a), 6):
        j = slice(i, i + 6)
        if ext.gemm_tc_multi(a[j], b[j], out[j], flip[j], [alpha] * len(a[j]), a_mn, 0, True):
            _native_mod._count()
            continue
        for x, y, o, t in zip(a[j], b[j], out[j], flip[j]):
            gemm(y, x, a_mn=True, b_mn=True, alpha=alpha, out=o) if t else gemm(x, y, a_mn=a_mn, b_mn=True, alpha=alpha, out=o)


def _adapter_grads(factors, inputs, r):
    """``dy_i^T t_i`` [N_i, r_i] for every (dy_i, t_i) of ``factors`` and ``t'_j^T x_j`` [r_j, K_j] for every (t'_j, x_j) of ``inputs``, of adapters
    whose largest rank is ``r``."""
    if not _narrow(r):
        return [gemm(dy, t, a_mn=True, b_mn=True) for dy, t in factors], [gemm(t, x, a_mn=True, b_mn=True) for t, x in inputs]
    a, b = [dy for dy, _ in factors] + [x for _, x in inputs], [t for _, t in factors] + [t for t, _ in inputs]
    out = [dy.new_empty(dy.shape[1], t.shape[1]) for dy, t in factors] + [x.new_empty(t.shape[1], x.shape[1]) for t, x in inputs]
    _multi(a, b, out, [False] * len(factors) + [True] * len(inputs), 1.0, True)
    return out[:len(factors)], out[len(factors):]


def _group_backward(gs, x2, t_cat, a_cat, ws, Bs, s, need_x, more_factors=(), more_inputs=()):
    """Gradients of a group of LoRA projections of ``x2``: (d x | None, d [A_1; ..; A_n], [d B_i], those of further pairs as _adapter_grads takes them)."""
    n, r = len(gs), t_cat.shape[1] // len(gs)
    tp_cat = torch.empty(x2.shape[0], n * r, dtype=x2.dtype, device=x2.device)
    tps = [tp_cat[:, i * r:(i + 1) * r] for i in range(n)]                                      # t'_i = s dy_i B_i
    if _narrow(r):
        _multi(list(gs), list(Bs), tps, [False] * n, s, False)
    else:
        for g, b, tp in zip(gs, Bs, tps):
            gemm(g, b, b_mn=True, alpha=s, out=tp)
    gx = sum_gemms([*gs, tp_cat], [*ws, a_cat]) if need_x else None                           # sum_i dy_i W_i + [t'_1 .. t'_n] [A_1; ..; A_n]
    gbs, gas = _adapter_grads([(gs[i], t_cat[:, i * r:(i + 1) * r]) for i in range(n)] + list(more_factors), [(tp_cat, x2)] + list(more_inputs),
                              max([r] + [t.shape[1] for _, t in more_factors]))
    return gx, gas[0], gbs[:n], gbs[n:] + gas[1:]


def _projections(x2, ws, bs, ts=(), Bs=()):
    """``x2 W_i^T + t_i B_i^T + b_i`` for every i, in one launch where four or fewer of them have aligned biases; their sums are those of their own GEMMs."""
    if 1 < len(ws) <= 4 and all(b is None or (b.is_contiguous() and b.dtype == torch.bfloat16 and b.data_ptr() % 16 == 0) for b in bs):
        _native_mod._count()
        return _native_mod.ext().gemm_tc_cat(x2, list(ws), list(bs), list(ts), list(Bs))
    return [gemm(x2, w, a2=ts[i] if ts else None, b2=Bs[i] if Bs else None, bias=bs[i]) for i, w in enumerate(ws)]


class _LoraGroupFn(torch.autograd.Function):
    """Several LoRA projections of ONE input (q / k / v, gate / up): the rank-r down-projections share a launch
    (``t = s x [A_1; ...; A_n]^T``), the base GEMMs share another and take their slices of ``t`` as dual-source-K operands, and in the backward the
    gradients of all factors come out of one launch and ``dx`` out of one over all projections and the LoRA term.  Compared with
    n independent ``_LoraLinearFn``: n - 1 fewer skinny launches per direction, ``x`` is re-read once instead of n times."""

    @staticmethod
    def forward(ctx, x, scaling, n, *flat):
        x2 = _rows(x)
        ws, bs, As, Bs = flat[0::4], flat[1::4], flat[2::4], flat[3::4]
        r = As[0].shape[0]
        a_cat = torch.cat(As, 0)                                             # [n r, K]
        t_cat = gemm(x2, a_cat, alpha=scaling)                               # [T, n r]
        ys = _projections(x2, ws, bs, [t_cat[:, i * r:(i + 1) * r] for i in range(n)], Bs)
        ctx.save_for_backward(x2, t_cat, a_cat, *ws, *Bs)
        ctx.meta = (scaling, n, r, x.shape)
        return tuple(y.view(*x.shape[:-1], y.shape[-1]) for y in ys)

    @staticmethod
    def backward(ctx, *gys):
        s, n, r, xshape = ctx.meta
        saved = ctx.saved_tensors
        x2, t_cat, a_cat = saved[:3]
        ws, Bs = saved[3:3 + n], saved[3 + n:3 + 2 * n]
        gx, ga_cat, gbs, _ = _group_backward([_rows(g) for g in gys], x2, t_cat, a_cat, ws, Bs, s, ctx.needs_input_grad[0])
        grads = [gx.view(xshape) if gx is not None else None, None, None]
        for i in range(n):
            grads += [None, None, ga_cat[i * r:(i + 1) * r], gbs[i]]
        return tuple(grads)


class _LoraMlpFn(torch.autograd.Function):
    """``(silu(gate) * up) Wd^T`` with LoRA on all three projections, frozen bases without biases.  Forward: one GEMM leaves gate, up and their
    product.  Backward: the product's gradient is formed and taken apart into those of gate and up in one GEMM's epilogue and never stored."""

    @staticmethod
    def forward(ctx, x, scaling, wg, ag, bg, wu, au, bu, wd, ad, bd):
        x2, r, ext = _rows(x), ag.shape[0], _native_mod.ext()
        a_cat = torch.cat([ag, au], 0)
        t_cat = gemm(x2, a_cat, alpha=scaling)
        _native_mod._count()
        act, gate, up = ext.gemm_tc_swiglu_pair_keep(x2, wg, wu, t_cat[:, :r], t_cat[:, r:], bg, bu)
        td = gemm(act, ad, alpha=scaling)
        y = gemm(act, wd, a2=td, b2=bd)
        ctx.save_for_backward(x2, t_cat, a_cat, wg, wu, bg, bu, gate, up, act, wd, ad, bd, td)
        ctx.meta = (scaling, r, x.shape)
        return y.view(*x.shape[:-1], y.shape[-1])

    @staticmethod
    def backward(ctx, gy):
        s, r, xshape = ctx.meta
        x2, t_cat, a_cat, wg, wu, bg, bu, gate, up, act, wd, ad, bd, td = ctx.saved_tensors
        g2 = _rows(gy)
        tpd = gemm(g2, bd, b_mn=True, alpha=s)                                                 # s dy Bd
        _native_mod._count()
        dgate, dup = _native_mod.ext().gemm_tc_dswiglu(g2, wd, tpd, ad, gate, up)
        gx, ga_cat, (gbg, gbu), (gbd, gad) = _group_backward([dgate, dup], x2, t_cat, a_cat, [wg, wu], [bg, bu], s, ctx.needs_input_grad[0], [(g2, td)], [(tpd, act)])
        return (gx.view(xshape) if gx is not None else None, None, None, ga_cat[:r], gbg, None, ga_cat[r:], gbu, None, gad, gbd)


def linear_add(x, w, residual, a=None, b=None, scaling: float = 0.0):
    """``residual + (x W^T + scaling (x A^T) B^T)`` without autograd, the sum in brackets rounded to bf16 as by its own GEMM; None where that GEMM does
    not apply."""
    if (x.numel() == 0 or not (supported(x, w) if a is None else lora_supported(x, w, a, b))
            or residual.dtype != torch.bfloat16 or residual.shape != (*x.shape[:-1], w.shape[0]) or residual.device != x.device):
        return None
    x2 = _rows(x)
    t = None if a is None else gemm(x2, a, alpha=scaling)
    return gemm(x2, w, a2=t, b2=b, residual=_rows(residual)).view(residual.shape)


def lora_mlp(x, gate, up, down, scaling: float):
    """``gate`` / ``up`` / ``down`` = (W, A, B); None when the fused form does not take the call."""
    (wg, ag, bg), (wu, au, bu), (wd, ad, bd) = gate, up, down
    if (x.numel() == 0 or wg.shape != wu.shape or wd.shape[1] != wg.shape[0] or ag.shape != au.shape or x.shape[-1] != wg.shape[1]
            or not (lora_supported(x, wg, ag, bg) and lora_supported(x, wu, au, bu)) or ad.shape[1] != wg.shape[0]
            or any(w.dtype != torch.bfloat16 or not w.is_contiguous() or any(n % 8 for n in w.shape) for w in (wd, ad, bd))):
        return None
    return _LoraMlpFn.apply(x, float(scaling), *gate, *up, *down)


def lora_linear_group(x, projs, scaling: float):
    """``projs``: [(W, bias | None, A, B), ...] sharing the input ``x`` -> list of outputs."""
    flat = []
    for w, bias, a, b in projs:
        flat += [w, bias, a, b]
    return list(_LoraGroupFn.apply(x, float(scaling), len(projs), *flat))


def swiglu_linears(x, gate, up, scaling: float = 0.0):
    """``silu(x Wg^T) * (x Wu^T)`` without the two projections in memory (no autograd).  Gate and up are rounded to bf16 before they are combined
    and summed in the order of their own GEMMs, so that the result is bit for bit that of ``swiglu_pair(x Wg^T, x Wu^T)``, which the training
    forward takes: log-probabilities of an unchanged policy have to agree.  ``gate`` / ``up`` = (W, A | None, B | None) with a LoRA term of
    ``scaling`` when A and B are given.  None when the fused GEMM does not take the call.  Two GEMMs and an activation pass against one, 1536 -> 8960
    features: 256 rows 28 / 17 us (with adapters 42 / 31), 1000 rows 57 / 41 (73 / 57), 32 768 rows 1602 / 1213 (1531 / 1295)."""
    (wg, ag, bg), (wu, au, bu) = gate, up
    x2 = _rows(x)
    if x2.shape[0] == 0 or not (supported(x, wg) and supported(x, wu)) or wg.shape != wu.shape or (ag is None) != (au is None):
        return None
    if ag is None:
        if _native_mod.ext().gemm_tc_auto_splits(x2.shape[0], *wg.shape, x2.get_device()) > 1:
            return None                                # their own GEMMs would add up ranges of the contraction: other sums
        _native_mod._count()
        y = _native_mod.ext().gemm_tc_swiglu_pair(x2, wg, wu)
    else:
        if ag.shape != au.shape or not (lora_supported(x, wg, ag, bg) and lora_supported(x, wu, au, bu)):
            return None
        r = ag.shape[0]
        t = gemm(x2, torch.cat([ag, au], 0), alpha=scaling)
        _native_mod._count()
        y = _native_mod.ext().gemm_tc_swiglu_pair(x2, wg, wu, t[:, :r], t[:, r:], bg, bu)
    return y.view(*x.shape[:-1], wg.shape[0])
