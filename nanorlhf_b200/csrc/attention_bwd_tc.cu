// tcgen05 / TMEM / TMA flash-attention BACKWARD (causal, packed varlen, GQA, head_dim 128) for sm_100a.
//
// Two kernels, no atomics (same decomposition as the mma.sync version in attention_varlen.cu, which stays the oracle); dK / dV and dQ are blocks of one:
//   delta   : delta[h, t] = sum_d dO * O                                   (half a warp per (token, head))
//   dK / dV : one CTA per (128-key block, kv head).  K_j, V_j stay in smem; the CTA streams (q head of the group,
//             64-row query block) pairs:   S^T = K_j Q_i^T,  dP^T = V_j dO_i^T          (tcgen05, TMEM lanes = keys)
//             P^T = exp2(S^T*c - lse_i),  dS^T = P^T o (dP^T - delta_i)                   (softmax warps, one key row each)
//             dV_j += P^T dO_i,  dK_j += dS^T Q_i                                         (tcgen05, accumulators in TMEM)
//   dQ      : one CTA per (128-row query block, q head).  Q_i, dO_i stay in smem; the CTA streams 64-key blocks:
//             S = Q_i K_j^T,  dP = dO_i V_j^T  ->  dS = P o (dP - delta)  ->  dQ_i += dS K_j
// (the scale of the scores is applied to the float accumulators of dK and dQ at the end).
// Shared structure: warp 0 = TMA producer (4-stage ring), warp 1 = single-thread MMA issuer, warps 2..17 = four
// elementwise warpgroups: two that share the columns of a block take alternate blocks (each pair owns one S/dP TMEM buffer), so
// the exp2/convert work of block n overlaps the MMAs of block n+1.  P and dS go back as bf16 into the TMEM columns of their S and dP and are the A
// operand of the next MMA from there.  The operands that must be read "transposed" (dO_i, Q_i for dV/dK; K_j for dQ) are
// consumed in place as MN-major UMMA operands - nothing is transposed in smem.
// Blocks start from the most work to the least over all sequences: a key block in front of a long sequence is up to a whole
// SM's share of the work, and one that starts late is waited for by the rest of the chip.
// Before (P and dS through shared memory, one warpgroup per block, blocks in the order of their position) each block waited for one warp per
// scheduler and the store's round trip, and the last key blocks of a launch ran alone: 28 heads over 4, 2 x 6005 tokens
// dK / dV 1672 -> 915 us, dQ 1130 -> 728 us (1.1 PFLOP/s).
// Replaces the flash-attn-2 backward the reference reaches through HF (attn_implementation="flash_attention_2",
// GRPO/grpo.py:219; training step GRPO/grpo_trainer.py:652).
#include "attention_tc.cuh"
#include "kernels.h"
#include "launch.h"

namespace nrl {

constexpr int kBwdThreads = 576;     // TMA, MMA, and four elementwise warpgroups: block parity x half of its columns
constexpr int kP128 = 128 * 128;     // [128 rows][64 x bf16] swizzled panel (16 KB)
constexpr int kT128 = 2 * kP128;     // 128 x 128 bf16 tile (32 KB)
constexpr int kP64 = 64 * 128;       // [64 rows][64 x bf16] panel (8 KB)
constexpr int kT64 = 2 * kP64;       // 64 x 128 bf16 tile (16 KB)
constexpr int kRing = 4;

struct AttnBwdParams {
  const int* cu_seqlens;
  const float* lse;           // [Hq, T]
  const float* delta;         // [Hq, T]
  __nv_bfloat16 *dq, *dk, *dv;
  long dq_stride_t, dkv_stride_t;
  int num_seqs, total_tokens, Hq, G;
  float scale, scale_log2;
};

// The `rank`-th block of 128 rows in the order of descending work: `level` counts the blocks of its sequence on the side where its work
// lies (behind it for keys, in front of it for queries).  Result through `info` (4 ints of shared memory).
NRL_DEVICE bool bwd_locate(const int* cu, int num_seqs, int rank, int* info, int& level, int& blocks, int& seq_start, int& seq_len) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int hi = 0, above = 0;                                     // blocks of the longest sequence; blocks with a level >= hi
    for (int s = lane; s < num_seqs; s += 32) hi = max(hi, (cu[s + 1] - cu[s] + 127) / 128);
    hi = __reduce_max_sync(0xffffffffu, hi);
    int lo = 0;
    bool found = rank < attn_blocks_from<128>(cu, num_seqs, 0, lane);
    while (found && hi - lo > 1) {
      const int mid = (lo + hi) >> 1, n = attn_blocks_from<128>(cu, num_seqs, mid, lane);
      if (rank < n) { lo = mid; } else { hi = mid; above = n; }
    }
    const int src = found ? attn_nth_sequence<128>(cu, num_seqs, lo, rank - above, lane) : 0;
    if (lane == 0) { info[0] = found; info[1] = lo; info[2] = cu[src]; info[3] = cu[src + 1] - cu[src]; }
  }
  __syncthreads();
  if (!info[0]) return false;
  level = info[1]; seq_start = info[2]; seq_len = info[3];
  blocks = (seq_len + 127) / 128;
  return true;
}

// 16 columns of one row: P = 2^(S * c - lse), dS = P (dP - delta) as bf16 pairs.  nl(i), nd(i): -lse and -delta of columns i, i + 1;
// MASK: columns without their bit in `see` are 0.
template <bool MASK, bool WANT_P, class NL, class ND>
NRL_DEVICE void bwd_chunk(const uint32_t (&sv)[16], const uint32_t (&dv)[16], uint64_t sc2, NL nl, ND nd, uint32_t see, uint32_t* pk,
                          uint32_t* dk) {
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float p0, p1, d0, d1;
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sc2, nl(i)), p0, p1);
    p0 = ex2_approx(p0);
    p1 = ex2_approx(p1);
    if (MASK) {
      if (!(see & (1u << i))) p0 = 0.f;
      if (!(see & (2u << i))) p1 = 0.f;
    }
    unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), add_f32x2(pack_f32x2(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1])), nd(i))), d0, d1);
    if (WANT_P) pk[i / 2] = pack_bf16x2(p0, p1);
    dk[i / 2] = pack_bf16x2(d0, d1);
  }
}

// Half a warp per pair, sixteen bytes per lane, two pairs in flight: 12 011 tokens x 28 heads 51 -> 29 us (8 bytes per lane, one pair per warp before)
__global__ void attn_bwd_delta_tc_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                         float* __restrict__ delta, long o_stride_t, int total, unsigned Hq, unsigned pairs) {
  pdl_wait();
  pdl_launch_dependents();
  const int sub = threadIdx.x & 15;
  const unsigned first = (blockIdx.x * (blockDim.x >> 4) + (threadIdx.x >> 4)) * 2;
  uint4 a[2], b[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const unsigned idx = min(first + u, pairs - 1), t = idx / Hq, h = idx - t * Hq;
    const long off = t * o_stride_t + h * 128 + sub * 8;
    a[u] = *reinterpret_cast<const uint4*>(o + off);
    b[u] = *reinterpret_cast<const uint4*>(dout + off);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, bw[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = unpack_bf16x2(aw[e]), y = unpack_bf16x2(bw[e]);
      acc = fmaf(x.x, y.x, fmaf(x.y, y.y, acc));
    }
#pragma unroll
    for (int m = 8; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    const unsigned idx = first + u, t = idx / Hq, h = idx - t * Hq;
    if (sub == 0 && idx < pairs) delta[static_cast<long>(h) * total + t] = acc;
  }
}

// =====================================================================================================================
// dK / dV
// =====================================================================================================================
struct DkdvSmem {
  static constexpr int kK = 0;
  static constexpr int kV = kT128;
  static constexpr int kQ = 2 * kT128;                     // ring
  static constexpr int kDO = kQ + kRing * kT64;            // ring
  static constexpr int kLD = kDO + kRing * kT64;           // [wg][parity][-lse2 x 32 | -delta x 32] floats
  static constexpr int kBar = kLD + 4 * 2 * 64 * 4;
  static constexpr int kTotal = kBar + 256;
};

NRL_DEVICE void bwd_dkdv(uint8_t* smem, unsigned block, const CUtensorMap& tmQ, const CUtensorMap& tmDO, const CUtensorMap& tmK,
                         const CUtensorMap& tmV, const AttnBwdParams& p) {
  using L = DkdvSmem;
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* qdo_full = kv_full + 1;            // [kRing]
  uint64_t* qdo_empty = qdo_full + kRing;      // [kRing]
  uint64_t* s_full = qdo_empty + kRing;        // [parity]  S^T and dP^T of the block are in TMEM
  uint64_t* pds_ready = s_full + 2;            // [parity]  P^T / dS^T of the block have replaced them
  uint64_t* done_bar = pds_ready + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done_bar + 1);
  int* info = reinterpret_cast<int*>(tmem_ptr + 4);      // its own 16-byte slot: tcgen05.alloc writes next to it

  int behind, blocks, seq_start, seq_len;
  const int rank = block / (p.Hq / p.G), kvh = block - rank * (p.Hq / p.G);
  if (!bwd_locate(p.cu_seqlens, p.num_seqs, rank, info, behind, blocks, seq_start, seq_len)) return;
  const int kb = blocks - 1 - behind;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int key0 = kb * 128;
  const int i_begin = key0 / 64;                                   // first 64-row query block that sees these keys
  const int n_qb = (seq_len + 63) / 64 - i_begin;                  // >= 1
  const int n_iter = p.G * n_qb;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 1 && lane == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < kRing; ++i) { mbar_init(&qdo_full[i], 1); mbar_init(&qdo_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&pds_ready[i], 8); }
    mbar_init(done_bar, 1);
    fence_mbar_init();
  }
  if (warp == 1) { __syncwarp(); tmem_alloc(tmem_ptr, 512); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  pdl_launch_dependents();
  // TMEM columns: S^T[parity] 0/64, dP^T[parity] 128/192, dV 256..383, dK 384..511

  if (warp == 0) {
    // ============================== TMA producer ==============================
    if (elect_one()) {
      mbar_arrive_expect_tx(kv_full, 2 * kT128);
      tma_load_2d(smem + L::kK, &tmK, kv_full, kvh * 128, seq_start + key0);
      tma_load_2d(smem + L::kK + kP128, &tmK, kv_full, kvh * 128 + 64, seq_start + key0);
      tma_load_2d(smem + L::kV, &tmV, kv_full, kvh * 128, seq_start + key0);
      tma_load_2d(smem + L::kV + kP128, &tmV, kv_full, kvh * 128 + 64, seq_start + key0);
      int st = 0;
      uint32_t phase = 0;
      int head = kvh * p.G, qi = 0;
      for (int it = 0; it < n_iter; ++it) {
        const int row = seq_start + (i_begin + qi) * 64;
        mbar_wait(&qdo_empty[st], phase ^ 1);
        mbar_arrive_expect_tx(&qdo_full[st], 2 * kT64);
        uint8_t* sq = smem + L::kQ + st * kT64;
        uint8_t* sd = smem + L::kDO + st * kT64;
        tma_load_2d(sq, &tmQ, &qdo_full[st], head * 128, row);
        tma_load_2d(sq + kP64, &tmQ, &qdo_full[st], head * 128 + 64, row);
        tma_load_2d(sd, &tmDO, &qdo_full[st], head * 128, row);
        tma_load_2d(sd + kP64, &tmDO, &qdo_full[st], head * 128 + 64, row);
        if (++qi == n_qb) { qi = 0; ++head; }
        if (++st == kRing) { st = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ============================== MMA issuer ==============================
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc(128, 64, 1, 1);          // [128 keys] x [64 q], both K-major (over d)
      constexpr uint32_t idesc_g = make_idesc_bmn(128, 128);          // [128 keys] x [128 d], B MN-major (over q)
      const uint32_t k_addr = smem_u32(smem + L::kK), v_addr = smem_u32(smem + L::kV);
      mbar_wait(kv_full, 0);
      tc_fence_after();
      int st_s = 0;
      uint32_t ph_s = 0;
      auto issue_sdp = [&](int it) {
        const int b = it & 1;
        mbar_wait(&qdo_full[st_s], ph_s);
        tc_fence_after();
        const uint32_t q_addr = smem_u32(smem + L::kQ + st_s * kT64);
        const uint32_t do_addr = smem_u32(smem + L::kDO + st_s * kT64);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16(tmem_base + b * 64, make_smem_desc_sw128(k_addr + (k >> 2) * kP128 + (k & 3) * 32),
                   make_smem_desc_sw128(q_addr + (k >> 2) * kP64 + (k & 3) * 32), idesc_s, k != 0 ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16(tmem_base + 128 + b * 64, make_smem_desc_sw128(v_addr + (k >> 2) * kP128 + (k & 3) * 32),
                   make_smem_desc_sw128(do_addr + (k >> 2) * kP64 + (k & 3) * 32), idesc_s, k != 0 ? 1u : 0u);
        umma_commit(&s_full[b]);
        if (++st_s == kRing) { st_s = 0; ph_s ^= 1; }
      };
      issue_sdp(0);
      int st = 0;
      for (int it = 0; it < n_iter; ++it) {
        const int b = it & 1;
        if (it + 1 < n_iter) issue_sdp(it + 1);             // overlaps the elementwise work of block it
        mbar_wait(&pds_ready[b], (it >> 1) & 1);
        tc_fence_after();
        const uint32_t q_addr = smem_u32(smem + L::kQ + st * kT64);
        const uint32_t do_addr = smem_u32(smem + L::kDO + st * kT64);
#pragma unroll
        for (int k = 0; k < 4; ++k)            // 4 x 16 query rows
          umma_f16_ts(tmem_base + 256, tmem_base + b * 64 + (k >> 1) * 32 + (k & 1) * 8, make_smem_desc_sw128_mn(do_addr + k * 16 * 128, kP64), idesc_g,
                      (it | k) != 0 ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16_ts(tmem_base + 384, tmem_base + 128 + b * 64 + (k >> 1) * 32 + (k & 1) * 8, make_smem_desc_sw128_mn(q_addr + k * 16 * 128, kP64), idesc_g,
                      (it | k) != 0 ? 1u : 0u);
        umma_commit(&qdo_empty[st]);
        if (++st == kRing) st = 0;
      }
      umma_commit(done_bar);
    }
    __syncwarp();
  } else {
    // ============================== elementwise warpgroups ==============================
    const int wg = (warp - 2) >> 2, par = wg & 1, half = wg >> 1;        // blocks of one parity, 32 of their 64 query columns
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                          // key row in tile == TMEM lane
    const int t128 = (warp - 2 - wg * 4) * 32 + lane;        // 0..127 within the warpgroup
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const int kk = key0 + r;
    float* ld_base = reinterpret_cast<float*>(smem + L::kLD) + wg * 128;
    int head = kvh * p.G, qi = par;                          // of the block that is fetched next
    auto load_ld = [&](int it) -> float {
      // threads 0..31 fetch -lse (in log2 units), 32..63 fetch -delta, of the columns' query rows of block `it`
      if (it >= n_iter || t128 >= 64) return 0.f;
      const int qq = (i_begin + qi) * 64 + half * 32 + (t128 & 31);
      if (qq >= seq_len) return t128 < 32 ? -INFINITY : 0.f;         // lse = +inf  =>  P = 0 for rows past the end
      const long off = static_cast<long>(head) * p.total_tokens + seq_start + qq;
      return t128 < 32 ? p.lse[off] * -1.4426950408889634f : -p.delta[off];
    };
    const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2);
    const uint32_t t_s = tmem_base + par * 64 + half * 32 + lane_off, t_dp = t_s + 128;
    while (qi >= n_qb) { qi -= n_qb; ++head; }
    float ld_next = load_ld(par);
    for (int it = par; it < n_iter; it += 2) {
      const int n = it >> 1;
      float* ldbuf = ld_base + (n & 1) * 64;
      if (t128 < 64) ldbuf[t128] = ld_next;
      const int q0 = (i_begin + qi) * 64 + half * 32;
      named_barrier_sync(1 + wg, 128);
      for (qi += 2; qi >= n_qb; qi -= n_qb) ++head;
      ld_next = load_ld(it + 2);
      mbar_wait(&s_full[par], n & 1);
      tc_fence_after();
      uint32_t pk[16], dk[16];
      const uint64_t* ld = reinterpret_cast<const uint64_t*>(ldbuf);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sv[16], dv[16];
        tmem_ld_32x32b_x16(t_s + c * 16, sv);
        tmem_ld_32x32b_x16(t_dp + c * 16, dv);
        tmem_ld_wait();
        auto nl = [&](int i) { return ld[c * 8 + i / 2]; };
        auto nd = [&](int i) { return ld[16 + c * 8 + i / 2]; };
        if (q0 < key0 + 127) bwd_chunk<true, true>(sv, dv, sc2, nl, nd, mask_from(kk - q0 - c * 16), pk + c * 8, dk + c * 8);
        else bwd_chunk<false, true>(sv, dv, sc2, nl, nd, 0u, pk + c * 8, dk + c * 8);
      }
      tmem_st_32x32b_x16(t_s, pk);
      tmem_st_32x32b_x16(t_dp, dk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_ready[par]);
    }
    // ---- epilogue: parity 0 writes dV, parity 1 writes dK, each warpgroup 64 columns ----
    mbar_wait(done_bar, 0);
    tc_fence_after();
    const bool row_ok = kk < seq_len;
    const float f = par == 0 ? 1.f : p.scale;
    __nv_bfloat16* dst = (par == 0 ? p.dv : p.dk) + static_cast<long>(seq_start + kk) * p.dkv_stride_t + kvh * 128 + half * 64;
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
      uint32_t ov[32];
      tmem_ld_32x32b_x32(tmem_base + 256 + par * 128 + half * 64 + c * 32 + lane_off, ov);     // warp-converged (.sync.aligned)
      tmem_ld_wait();
      if (row_ok) {
#pragma unroll
        for (int i = 0; i < 16; ++i) ov[i] = pack_bf16x2(__uint_as_float(ov[2 * i]) * f, __uint_as_float(ov[2 * i + 1]) * f);
        stg_v8(dst + c * 32, ov);
        stg_v8(dst + c * 32 + 16, ov + 8);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// =====================================================================================================================
// dQ
// =====================================================================================================================
struct DqSmem {
  static constexpr int kQ = 0;
  static constexpr int kDO = kT128;
  static constexpr int kK = 2 * kT128;                     // ring
  static constexpr int kV = kK + kRing * kT64;             // ring
  static constexpr int kBar = kV + kRing * kT64;
  static constexpr int kTotal = kBar + 256;
};

NRL_DEVICE void bwd_dq(uint8_t* smem, unsigned block, const CUtensorMap& tmQ, const CUtensorMap& tmDO, const CUtensorMap& tmK,
                       const CUtensorMap& tmV, const AttnBwdParams& p) {
  using L = DqSmem;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* kv_full = q_full + 1;              // [kRing]
  uint64_t* kv_empty = kv_full + kRing;        // [kRing]
  uint64_t* s_full = kv_empty + kRing;         // [wg]
  uint64_t* ds_ready = s_full + 2;             // [wg]
  uint64_t* done_bar = ds_ready + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done_bar + 1);
  int* info = reinterpret_cast<int*>(tmem_ptr + 4);      // its own 16-byte slot: tcgen05.alloc writes next to it

  int mb, blocks, seq_start, seq_len;
  const int rank = block / p.Hq, head = block - rank * p.Hq, kvh = head / p.G;
  if (!bwd_locate(p.cu_seqlens, p.num_seqs, rank, info, mb, blocks, seq_start, seq_len)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q0 = mb * 128;
  const int n_kb = min((seq_len + 63) / 64, (q0 + 128 + 63) / 64);

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 1 && lane == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < kRing; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&ds_ready[i], 8); }
    mbar_init(done_bar, 1);
    fence_mbar_init();
  }
  if (warp == 1) { __syncwarp(); tmem_alloc(tmem_ptr, 512); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  pdl_launch_dependents();
  // TMEM columns: S[parity] 0/64, dP[parity] 128/192, dQ 256..383

  if (warp == 0) {
    if (elect_one()) {
      mbar_arrive_expect_tx(q_full, 2 * kT128);
      tma_load_2d(smem + L::kQ, &tmQ, q_full, head * 128, seq_start + q0);
      tma_load_2d(smem + L::kQ + kP128, &tmQ, q_full, head * 128 + 64, seq_start + q0);
      tma_load_2d(smem + L::kDO, &tmDO, q_full, head * 128, seq_start + q0);
      tma_load_2d(smem + L::kDO + kP128, &tmDO, q_full, head * 128 + 64, seq_start + q0);
      int st = 0;
      uint32_t phase = 0;
      for (int j = 0; j < n_kb; ++j) {
        mbar_wait(&kv_empty[st], phase ^ 1);
        mbar_arrive_expect_tx(&kv_full[st], 2 * kT64);
        uint8_t* sk = smem + L::kK + st * kT64;
        uint8_t* sv = smem + L::kV + st * kT64;
        const int row = seq_start + j * 64;
        tma_load_2d(sk, &tmK, &kv_full[st], kvh * 128, row);
        tma_load_2d(sk + kP64, &tmK, &kv_full[st], kvh * 128 + 64, row);
        tma_load_2d(sv, &tmV, &kv_full[st], kvh * 128, row);
        tma_load_2d(sv + kP64, &tmV, &kv_full[st], kvh * 128 + 64, row);
        if (++st == kRing) { st = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc(128, 64, 1, 1);          // [128 q] x [64 keys], both K-major (over d)
      constexpr uint32_t idesc_g = make_idesc_bmn(128, 128);          // [128 q] x [128 d], B = K_j MN-major (over keys)
      const uint32_t q_addr = smem_u32(smem + L::kQ), do_addr = smem_u32(smem + L::kDO);
      mbar_wait(q_full, 0);
      tc_fence_after();
      int st_s = 0;
      uint32_t ph_s = 0;
      auto issue_sdp = [&](int j) {
        const int b = j & 1;
        mbar_wait(&kv_full[st_s], ph_s);
        tc_fence_after();
        const uint32_t k_addr = smem_u32(smem + L::kK + st_s * kT64);
        const uint32_t v_addr = smem_u32(smem + L::kV + st_s * kT64);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16(tmem_base + b * 64, make_smem_desc_sw128(q_addr + (k >> 2) * kP128 + (k & 3) * 32),
                   make_smem_desc_sw128(k_addr + (k >> 2) * kP64 + (k & 3) * 32), idesc_s, k != 0 ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16(tmem_base + 128 + b * 64, make_smem_desc_sw128(do_addr + (k >> 2) * kP128 + (k & 3) * 32),
                   make_smem_desc_sw128(v_addr + (k >> 2) * kP64 + (k & 3) * 32), idesc_s, k != 0 ? 1u : 0u);
        umma_commit(&s_full[b]);
        if (++st_s == kRing) { st_s = 0; ph_s ^= 1; }
      };
      issue_sdp(0);
      int st = 0;
      for (int j = 0; j < n_kb; ++j) {
        const int b = j & 1;
        if (j + 1 < n_kb) issue_sdp(j + 1);
        mbar_wait(&ds_ready[b], (j >> 1) & 1);
        tc_fence_after();
        const uint32_t k_addr = smem_u32(smem + L::kK + st * kT64);
#pragma unroll
        for (int k = 0; k < 4; ++k)            // 4 x 16 keys
          umma_f16_ts(tmem_base + 256, tmem_base + 128 + b * 64 + (k >> 1) * 32 + (k & 1) * 8, make_smem_desc_sw128_mn(k_addr + k * 16 * 128, kP64), idesc_g,
                      (j | k) != 0 ? 1u : 0u);
        umma_commit(&kv_empty[st]);
        if (++st == kRing) st = 0;
      }
      umma_commit(done_bar);
    }
    __syncwarp();
  } else {
    const int wg = (warp - 2) >> 2, par = wg & 1, half = wg >> 1;        // blocks of one parity, 32 of their 64 keys
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                          // query row in tile == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const int row = q0 + r;
    const bool row_ok = row < seq_len;
    const long loff = static_cast<long>(head) * p.total_tokens + seq_start + row;
    const float lse2 = row_ok ? p.lse[loff] * 1.4426950408889634f : INFINITY;     // +inf => P = 0
    const float dl = row_ok ? p.delta[loff] : 0.f;
    const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2), nl2 = pack_f32x2(-lse2, -lse2), nd2 = pack_f32x2(-dl, -dl);
    const uint32_t t_s = tmem_base + par * 64 + half * 32 + lane_off, t_dp = t_s + 128;
    auto nl = [&](int) { return nl2; };
    auto nd = [&](int) { return nd2; };
    for (int j = par; j < n_kb; j += 2) {
      const int n = j >> 1;
      const int key0 = j * 64 + half * 32;
      const int hi = min(row, seq_len - 1) - key0;             // last visible key of these columns
      mbar_wait(&s_full[par], n & 1);
      tc_fence_after();
      uint32_t dk[16];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sv[16], dv[16];
        tmem_ld_32x32b_x16(t_s + c * 16, sv);
        tmem_ld_32x32b_x16(t_dp + c * 16, dv);
        tmem_ld_wait();
        if (key0 + 31 > q0 || key0 + 32 > seq_len) bwd_chunk<true, false>(sv, dv, sc2, nl, nd, ~mask_from(hi + 1 - c * 16), nullptr, dk + c * 8);
        else bwd_chunk<false, false>(sv, dv, sc2, nl, nd, 0u, nullptr, dk + c * 8);
      }
      tmem_st_32x32b_x16(t_dp, dk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_ready[par]);
    }
    // ---- epilogue: each warpgroup writes 32 of the 128 dQ columns ----
    mbar_wait(done_bar, 0);
    tc_fence_after();
    __nv_bfloat16* dst = p.dq + static_cast<long>(seq_start + row) * p.dq_stride_t + head * 128 + wg * 32;
    uint32_t ov[32];
    tmem_ld_32x32b_x32(tmem_base + 256 + wg * 32 + lane_off, ov);
    tmem_ld_wait();
    if (row_ok) {
#pragma unroll
      for (int i = 0; i < 16; ++i) ov[i] = pack_bf16x2(__uint_as_float(ov[2 * i]) * p.scale, __uint_as_float(ov[2 * i + 1]) * p.scale);
      stg_v8(dst, ov);
      stg_v8(dst + 16, ov + 8);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// Both in one launch, dQ's blocks behind those of dK / dV: neither takes anything from the other, and with two key heads dK / dV has a block for two SMs in
// three only, so that dQ starts on the SMs that it leaves idle.  us of the whole backward as launches one after the other / so: 4 sequences, 6601 tokens, 12
// heads over 2 250 / 164; 6 of 500, 28 over 4 116 / 76; 2 of 6005 1755 / 1582 to 1688; 4 of 6000 3529 / 3400; one of 300, 12 over 2 58 / 40.
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ64, const __grid_constant__ CUtensorMap tmDO64, const __grid_constant__ CUtensorMap tmK128,
                   const __grid_constant__ CUtensorMap tmV128, const __grid_constant__ CUtensorMap tmQ128, const __grid_constant__ CUtensorMap tmDO128,
                   const __grid_constant__ CUtensorMap tmK64, const __grid_constant__ CUtensorMap tmV64, const __grid_constant__ AttnBwdParams p,
                   const unsigned dkdv_blocks) {
  extern __shared__ __align__(1024) uint8_t smem[];
  pdl_wait();
  if (blockIdx.x < dkdv_blocks) bwd_dkdv(smem, blockIdx.x, tmQ64, tmDO64, tmK128, tmV128, p);
  else bwd_dq(smem, blockIdx.x - dkdv_blocks, tmQ128, tmDO128, tmK64, tmV64, p);
}

}  // namespace nrl

// maps: [0] Q box 64 rows, [1] dO box 64 rows, [2] K box 128 rows, [3] V box 128 rows  (dK / dV)
//       [4] Q box 128 rows, [5] dO box 128 rows, [6] K box 64 rows, [7] V box 64 rows  (dQ)
extern "C" cudaError_t nrl_attn_bwd_tc(const CUtensorMap* maps, const void* o, const void* dout, const float* lse,
                                       float* delta, void* dq, void* dk, void* dv, long o_stride_t, long dq_stride_t,
                                       long dkv_stride_t, const int* cu, int num_seqs, int total, int Hq, int Hkv,
                                       float scale, cudaStream_t s) {
  using namespace nrl;
  if (total == 0) return cudaSuccess;
  constexpr int smem = DkdvSmem::kTotal > DqSmem::kTotal ? DkdvSmem::kTotal : DqSmem::kTotal;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  const unsigned pairs = static_cast<unsigned>(total) * Hq;                   // O alone would be a terabyte at 2^32
  launch_dependent(attn_bwd_delta_tc_kernel, (pairs + 31) / 32, 256, 0, s, static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(dout), delta,
                   o_stride_t, total, Hq, pairs);
  AttnBwdParams p;
  p.cu_seqlens = cu; p.lse = lse; p.delta = delta;
  p.dq = static_cast<__nv_bfloat16*>(dq); p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv);
  p.dq_stride_t = dq_stride_t; p.dkv_stride_t = dkv_stride_t;
  p.num_seqs = num_seqs; p.total_tokens = total; p.Hq = Hq; p.G = Hq / Hkv;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  const unsigned most = total / 128 + num_seqs, grid_kv = most * Hkv, grid_q = most * Hq;
  launch_dependent(attn_bwd_tc_kernel, grid_kv + grid_q, kBwdThreads, smem, s, maps[0], maps[1], maps[2], maps[3], maps[4], maps[5], maps[6], maps[7], p,
                   grid_kv);
  return cudaGetLastError();
}
