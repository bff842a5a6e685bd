"""Tiny driver for `ncu --set full`: one launch each of the headline kernels at bench shapes."""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from nanorlhf_b200.ops import native  # noqa: E402

native.load()
dev = "cuda"
which = sys.argv[1] if len(sys.argv) > 1 else "all"
torch.manual_seed(0)
if which in ("all", "gemm"):
    a = torch.randn(2048, 1536, device=dev, dtype=torch.bfloat16)
    b = torch.randn(17920, 1536, device=dev, dtype=torch.bfloat16)
    for _ in range(3):
        native.gemm_bf16(a, b)
if which in ("all", "lmhead"):
    h = torch.randn(8192, 1536, device=dev, dtype=torch.bfloat16)
    w = (torch.randn(151936, 1536, device=dev) * 0.02).bfloat16()
    t = torch.randint(0, 151936, (8192,), device=dev, dtype=torch.int32)
    for _ in range(2):
        native.ext().lmhead_logprob_fwd(h, w, t, 1 / 0.9, 0)
if which in ("all", "decode"):
    S, ctx, Hq, Hkv, D = 2048, 1000, 12, 2, 128
    per = ctx // 16 + 1
    kc = torch.randn(S * per, Hkv, 16, D, device=dev, dtype=torch.bfloat16)
    vc = torch.randn_like(kc)
    bt = torch.arange(S * per, device=dev, dtype=torch.int32).view(S, per)
    cl = torch.full((S,), ctx, device=dev, dtype=torch.int32)
    q = torch.randn(S, Hq, D, device=dev, dtype=torch.bfloat16)
    for _ in range(3):
        native.paged_decode(q, kc, vc, bt, cl)
if which in ("all", "attn"):
    T = 4 * 1650
    cu = torch.tensor([0, 1650, 3300, 4950, 6600], device=dev, dtype=torch.int32)
    q = torch.randn(T, 12, 128, device=dev, dtype=torch.bfloat16)
    k = torch.randn(T, 2, 128, device=dev, dtype=torch.bfloat16)
    v = torch.randn(T, 2, 128, device=dev, dtype=torch.bfloat16)
    for _ in range(2):
        native.ext().attn_varlen_fwd(q, k, v, cu, 1650, 1 / math.sqrt(128), True)
if which in ("all", "deberta"):
    from nanorlhf_b200.models.deberta_v3 import build_bucket_lut
    lens = [1660] * 8
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device=dev, dtype=torch.int32)
    T = sum(lens)
    q = torch.randn(T, 16, 64, device=dev, dtype=torch.bfloat16)
    k = torch.randn(T, 16, 64, device=dev, dtype=torch.bfloat16)
    v = torch.randn(T, 16, 64, device=dev, dtype=torch.bfloat16)
    ra = torch.randn(16, T, 512, device=dev, dtype=torch.bfloat16)
    rb = torch.randn(16, T, 512, device=dev, dtype=torch.bfloat16)
    lut = build_bucket_lut(1660, 256, 512, 256, dev)
    for _ in range(2):
        native.ext().attn_varlen_fwd(q, k, v, cu, 1660, 1 / math.sqrt(192), False, ra, rb, lut)
if which in ("all", "attn_tc"):
    lens = [4096] * 4
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device=dev, dtype=torch.int32)
    T = sum(lens)
    q = torch.randn(T, 12, 128, device=dev, dtype=torch.bfloat16)
    k = torch.randn(T, 2, 128, device=dev, dtype=torch.bfloat16)
    v = torch.randn(T, 2, 128, device=dev, dtype=torch.bfloat16)
    for _ in range(2):
        o, lse = native.ext().attn_fwd_tc(q, k, v, cu, 1 / math.sqrt(128))
    native.ext().attn_bwd_tc(torch.randn_like(o), q, k, v, o, lse, cu, 1 / math.sqrt(128))
if which in ("all", "gemm_tc_ffn1", "gemm_tc_gate", "gemm_tc_dgrad", "gemm_tc_wgrad"):
    shapes = {"gemm_tc_ffn1": (26560, 4096, 1024, False, False), "gemm_tc_gate": (6912, 8960, 1536, False, False),
              "gemm_tc_dgrad": (6912, 1536, 8960, False, True), "gemm_tc_wgrad": (8960, 64, 6912, True, True)}
    for name, (M, N, K, amn, bmn) in shapes.items():
        if which not in ("all", name):
            continue
        a = torch.randn((K, M) if amn else (M, K), device=dev, dtype=torch.bfloat16)
        b = torch.randn((K, N) if bmn else (N, K), device=dev, dtype=torch.bfloat16)
        for _ in range(3):
            native.ext().gemm_tc(a, b, amn, bmn)
if which in ("all", "decode_fp8"):
    S, ctx, Hq, Hkv, D = 1024, 1000, 12, 2, 128
    per = ctx // 16 + 1
    kq = torch.randint(0, 120, (S * per, Hkv, 16, D), device=dev, dtype=torch.uint8)
    vq = torch.randint(0, 120, (S * per, Hkv, D, 16), device=dev, dtype=torch.uint8)
    ks = torch.rand(S * per, Hkv, 16, device=dev) * 0.01 + 0.001
    vs = torch.rand(S * per, Hkv, 16, device=dev) * 0.01 + 0.001
    bt = torch.arange(S * per, device=dev, dtype=torch.int32).view(S, per)
    cl = torch.full((S,), ctx, device=dev, dtype=torch.int32)
    q = torch.randn(S, Hq, D, device=dev, dtype=torch.bfloat16)
    for _ in range(3):
        native.ext().paged_decode_fp8(q, kq, vq, ks, vs, bt, cl, 1 / math.sqrt(D), 1)
if which in ("all", "sample", "sample_stream"):
    logits = torch.randn(1024, 151936, device=dev, dtype=torch.bfloat16)
    rid = torch.arange(1024, device=dev, dtype=torch.int32)
    for _ in range(3):                       # "sample": the cluster / shared-memory kernel; "sample_stream": the streaming fallback
        native.sample(logits, 0.9, 0.95, 1, 0, rid, rid, impl=1 if which == "sample_stream" else 0)
if which in ("all", "deberta_tma"):
    from nanorlhf_b200.models.deberta_v3 import build_bucket_lut
    lens = [1660] * 8
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device=dev, dtype=torch.int32)
    T = sum(lens)
    q, k, v = (torch.randn(T, 16, 64, device=dev, dtype=torch.bfloat16) for _ in range(3))
    ra, rb = (torch.randn(16, T, 512, device=dev, dtype=torch.bfloat16) for _ in range(2))
    lut = build_bucket_lut(1660, 256, 512, 256, dev)
    for _ in range(3):
        native.ext().deberta_attn_fwd(q, k, v, cu, 1660, 1 / math.sqrt(192), ra, rb, lut)
if which in ("all", "deberta_tc"):
    from nanorlhf_b200.models.deberta_v3 import build_bucket_lut
    lens = [1536] * 4
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device=dev, dtype=torch.int32)
    T = sum(lens)
    q, k, v = (torch.randn(T, 16, 64, device=dev, dtype=torch.bfloat16) for _ in range(3))
    pos_k = torch.randn(512, 16, 64, device=dev, dtype=torch.bfloat16).transpose(0, 1)
    rb = torch.randn(16, T, 512, device=dev, dtype=torch.bfloat16)
    lut = build_bucket_lut(1536, 256, 512, 256, dev)
    for _ in range(3):
        native.ext().deberta_attn_tc(q, k, v, cu, 1536, 1 / math.sqrt(192), pos_k, rb, lut)
if which in ("all", "gemm_tc_cut"):
    a, b = torch.randn(128, 8960, device=dev, dtype=torch.bfloat16), torch.randn(1536, 8960, device=dev, dtype=torch.bfloat16)
    for _ in range(3):                       # the ranges of a tile are a cluster
        native.ext().gemm_tc(a, b, False, False)
if which in ("all", "delta_chunk"):
    from types import SimpleNamespace
    from nanorlhf_b200.ops import hybrid
    E, n, H, D = 16, 512, 16, 128
    qkv = torch.randn(E * n, 3 * H * D, device=dev) * 0.1
    beta, decay = torch.rand(E * n, H, device=dev), torch.rand(E * n, H, device=dev) * 0.1 + 0.9
    plan = SimpleNamespace(cu=torch.arange(E + 1, device=dev, dtype=torch.int32) * n, start=torch.zeros(E, device=dev, dtype=torch.int32),
                           state_slot=torch.arange(E, device=dev, dtype=torch.int32))
    state, o = torch.zeros(E, H, D, D, device=dev), torch.empty(E * n, H * D, device=dev)
    for _ in range(3):
        hybrid.delta_scan(qkv, H * D, 2 * H * D, beta, decay, state, o, plan, H, False, impl="chunked")
if which in ("all", "dlogits"):
    h = torch.randn(8192, 1536, device=dev, dtype=torch.bfloat16)
    w = (torch.randn(151936, 1536, device=dev) * 0.02).bfloat16()
    t = torch.randint(0, 151936, (8192,), device=dev, dtype=torch.int32)
    lse = torch.full((8192,), 12.0, device=dev)
    g = torch.randn(8192, device=dev)
    for _ in range(3):
        native.ext().lmhead_dlogits(h, w, t, lse, g, 1 / 0.9)
if which in ("all", "kar1"):
    n = 540_672_000 // 8
    G, P = torch.randn(n, device=dev).bfloat16(), torch.randn(n, device=dev).bfloat16()
    m, v = torch.zeros(n, device=dev), torch.zeros(n, device=dev)
    mw = P.float()
    for _ in range(3):                      # world = 1 instantiation of the P2P kernel: the HBM-side cost of K-AR
        native.ext().allreduce_adam([G.data_ptr()], [P.data_ptr()], 0, 0, m, v, 0, n, 0, 6e-6, 0.9, 0.999, 1e-8, 0.0, 1, 1.0, False, 592, mw)
if which in ("all", "rl"):
    B, T = 256, 1500
    nl, ol, adv, rl = (torch.randn(B, T, device=dev) for _ in range(4))
    mk = torch.rand(B, T, device=dev) > 0.1
    for _ in range(3):
        native.ext().policy_loss(nl, ol, adv, mk, rl, 0.2, 0.01)
        native.gae_scan(adv, nl, 1.0, 0.95)
if which in ("all", "gemm_tc_fp8"):
    x, w = torch.randn(1024, 1536, device=dev, dtype=torch.bfloat16), torch.randn(17920, 1536, device=dev, dtype=torch.bfloat16)
    xq, xs = native.ext().quant_rows_e4m3(x)
    wq, ws = native.ext().quant_rows_e4m3(w)
    for _ in range(3):
        native.ext().gemm_tc_fp8(xq, xs, wq, ws, None, True)
torch.cuda.synchronize()
