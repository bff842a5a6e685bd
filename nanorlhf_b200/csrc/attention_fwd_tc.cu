// tcgen05 / TMEM / TMA flash-attention FORWARD (causal, packed varlen, GQA, head_dim 128) for sm_100a.
//
// Work item: 256 query rows of one head as TWO 128-row tiles (A, B) that share one K/V ring, walking the keys in blocks of 128.
//   warp 0       TMA producer : Q tiles, then K_0, V_0, K_1, V_1 ... into a ring of four 32 KB tiles (128B-swizzled panels of 64 dims)
//   warp 1       MMA issuer   : S_X = Q_X K_j^T, then per block O_X += P_X V_j and at once the next S_X, tiles alternating, so that the
//                               tensor pipe works on one tile while the other is in its softmax
//   warp 2       finds the next item (which sequence, which rows) while the current one is computed, the first one during the set-up
//   warps 4..11  one thread per query row: scores from TMEM, mask, online softmax (attention_tc.cuh), P as bf16 back into TMEM over its
//                scores, where it is the A operand of P V; O / l and LSE at the end.  The next item's queries and first keys arrive meanwhile.
// One persistent CTA per SM (TMEM 512 columns, 193 KB of shared memory).  Items go from the most to the fewest key blocks over all
// sequences, heads varying fastest, and are dealt to the CTAs forwards and backwards in turn, so that their shares come out even.
// Tensor pipe and special-function unit (2^x) are each 56 % busy at 4 x 4096 tokens, 12 heads over 2: what is left is the hand-over between
// scores, softmax and P V of the two tiles (attention_tc.cuh).
// The earlier form (blocks of 64 keys, P through swizzled shared memory, a CTA per item) spent its time on the shared-memory round trip of
// P and between CTAs: 28 heads over 4, 2 x 6005 tokens 648 -> 467 us (1.1 PFLOP/s).
// Backward: attention_bwd_tc.cu.  Oracle: the mma.sync kernels in attention_varlen.cu.  Together they replace flash-attn-2
// (attn_implementation="flash_attention_2", GRPO/grpo.py:219) on the training, log-prob and prefill paths.
#include "attention_tc.cuh"
#include "kernels.h"
#include "launch.h"

namespace nrl {

constexpr int kTcBM = 256;                 // query rows per item (two tiles of 128)
constexpr int kTcSlots = 4;                // ring of K and V tiles

struct AttnTcParams {
  const int* cu_seqlens;
  __nv_bfloat16* out;
  float* lse;                 // [Hq, T_total]
  long o_stride_t;
  int num_seqs, total_tokens, Hq, G;
  float scale_log2;
};

struct AttnTcSmem {
  static constexpr int kQ = 0;                                   // 2 tiles
  static constexpr int kRing = 2 * kAtTile;                      // kTcSlots tiles
  static constexpr int kBar = kRing + kTcSlots * kAtTile;        // mbarriers, TMEM pointer
  static constexpr int kTab = kBar + 256;                        // two items: head (-1: none left), q0, first token, length
  static constexpr int kTotal = kTab + 2 * 16;
};

struct AttnItem {
  int head, q0, start, len;
  NRL_DEVICE int blocks(int x) const {     // key blocks that tile x walks; tile B may lie entirely behind the end of the sequence
    return q0 + x * 128 < len ? q0 / 128 + 1 + x : 0;
  }
};
NRL_DEVICE AttnItem attn_item(const uint8_t* smem, uint64_t* tab_full, uint32_t k) {
  mbar_wait(&tab_full[k & 1], (k >> 1) & 1);
  const volatile int* t = reinterpret_cast<const volatile int*>(smem + AttnTcSmem::kTab + (k & 1) * 16);
  return {t[0], t[1], t[2], t[3]};
}

__global__ void __launch_bounds__(kAtThreads, 1)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const AttnTcParams p) {
  using L = AttnTcSmem;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBar);      // [kTcSlots]
  uint64_t* empty = full + kTcSlots;           // [kTcSlots]
  uint64_t* q_full = empty + kTcSlots;         // [tile]
  uint64_t* q_empty = q_full + 2;              // [tile]
  uint64_t* s_full = q_empty + 2;              // [tile]
  uint64_t* p_ready = s_full + 2;              // [tile]
  uint64_t* o_done = p_ready + 2;              // [tile]
  uint64_t* tab_full = o_done + 2;             // [2]
  uint64_t* tab_empty = tab_full + 2;          // [2]
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tab_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int i = 0; i < kTcSlots; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&empty[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&q_full[i], 1);
        mbar_init(&q_empty[i], 1);
        mbar_init(&s_full[i], 1);
        mbar_init(&p_ready[i], 4);             // one arrive per softmax warp of the tile
        mbar_init(&o_done[i], 1);
        mbar_init(&tab_full[i], 1);
        mbar_init(&tab_empty[i], 10);          // producer, MMA issuer, eight softmax warps
      }
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_ptr, 512);
  }
  pdl_wait();
  // warp 2: the blocks of the longest sequence and the first item, while barriers and tensor memory are set up
  const int* cu = p.cu_seqlens;
  int level = 0, above = 0, upto = 0;                                // row blocks with an index > level, >= level
  auto item_of = [&](uint32_t k) {
    const int at = (k & 1) ? (k + 1) * gridDim.x - 1 - blockIdx.x : k * gridDim.x + blockIdx.x;
    const int rank = at / p.Hq;
    while (level > 0 && rank >= upto) {
      --level;
      above = upto;
      upto = attn_blocks_from<kTcBM>(cu, p.num_seqs, level, lane);
    }
    if (rank >= upto) return make_int4(-1, 0, 0, 0);
    const int src = attn_nth_sequence<kTcBM>(cu, p.num_seqs, level, rank - above, lane);
    return make_int4(at - rank * p.Hq, level * kTcBM, cu[src], cu[src + 1] - cu[src]);
  };
  int4 next = make_int4(-1, 0, 0, 0);
  if (warp == 2) {
    for (int s = lane; s < p.num_seqs; s += 32) level = max(level, (cu[s + 1] - cu[s] + kTcBM - 1) / kTcBM);
    level = __reduce_max_sync(0xffffffffu, level);
    next = item_of(0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  pdl_launch_dependents();

  if (warp < 4) {
    attn_regs_issue();
    if (warp == 0) {
      // ============================== TMA producer ==============================
      if (elect_one()) {
        int slot = 0;
        uint32_t phase = 0, n_q[2] = {0, 0};
        auto load = [&](const CUtensorMap* tm, int col, int row) {
          mbar_wait(&empty[slot], phase ^ 1);
          uint8_t* dst = smem + L::kRing + slot * kAtTile;
          mbar_arrive_expect_tx(&full[slot], kAtTile);
          tma_load_2d(dst, tm, &full[slot], col, row);
          tma_load_2d(dst + kAtPanel, tm, &full[slot], col + 64, row);
          if (++slot == kTcSlots) { slot = 0; phase ^= 1; }
        };
        for (uint32_t k = 0;; ++k) {
          const AttnItem it = attn_item(smem, tab_full, k);
          mbar_arrive(&tab_empty[k & 1]);
          if (it.head < 0) break;
          const int kvc = it.head / p.G * kAtD, n = max(it.blocks(0), it.blocks(1));
          for (int x = 0; x < 2; ++x) {
            if (it.blocks(x) == 0) continue;
            mbar_wait(&q_empty[x], (n_q[x] & 1) ^ 1);
            ++n_q[x];
            uint8_t* dst = smem + L::kQ + x * kAtTile;
            mbar_arrive_expect_tx(&q_full[x], kAtTile);
            tma_load_2d(dst, &tmQ, &q_full[x], it.head * kAtD, it.start + it.q0 + x * 128);
            tma_load_2d(dst + kAtPanel, &tmQ, &q_full[x], it.head * kAtD + 64, it.start + it.q0 + x * 128);
          }
          for (int j = 0; j < n; ++j) {
            load(&tmK, kvc, it.start + j * kAtBN);
            load(&tmV, kvc, it.start + j * kAtBN);
          }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ============================== MMA issuer ==============================
      // elect.sync (not `lane == 0`) lets the compiler prove single-thread execution; otherwise every tcgen05.mma is wrapped in an
      // ELECT/branch loop whose latency exceeds these short MMAs
      if (elect_one()) {
        int slot = 0;                            // ring slot of the next tile in load order
        uint32_t phase = 0, n_p[2] = {0, 0}, n_q[2] = {0, 0};
        auto ring_next = [&]() {
          if (++slot == kTcSlots) { slot = 0; phase ^= 1; }
        };
        const uint32_t q_addr = smem_u32(smem + L::kQ), ring = smem_u32(smem + L::kRing);
        for (uint32_t k = 0;; ++k) {
          const AttnItem it = attn_item(smem, tab_full, k);
          mbar_arrive(&tab_empty[k & 1]);
          if (it.head < 0) break;
          const int nx[2] = {it.blocks(0), it.blocks(1)}, n = max(nx[0], nx[1]);
          auto issue_s = [&](int x, int j, int s) {
            attn_issue_s(tmem_base + x * kAtBN, q_addr + x * kAtTile, ring + s * kAtTile);
            umma_commit(&s_full[x]);
            if (j == nx[x] - 1) umma_commit(&q_empty[x]);
          };
          mbar_wait(&full[slot], phase);
#pragma unroll
          for (int x = 0; x < 2; ++x)
            if (nx[x] > 0) {
              mbar_wait(&q_full[x], n_q[x] & 1);
              ++n_q[x];
              tc_fence_after();
              issue_s(x, 0, slot);
            }
          umma_commit(&empty[slot]);
          ring_next();
          for (int j = 0; j < n; ++j) {
            const int v_slot = slot;             // load order is K_0, V_0, K_1 ...: the next K sits behind this V
            mbar_wait(&full[v_slot], phase);
            ring_next();
            const int k_slot = slot;
            if (j + 1 < n) {
              mbar_wait(&full[k_slot], phase);
              ring_next();
            }
            // keys behind the end of the sequence belong to another one: their P is 0, and groups of 16 of them stay out.  The last group
            // may hold up to 15 rows of the next sequence's V times 0: an infinity or NaN there reaches this block's rows
            const int steps = min(8, (it.len - j * kAtBN + 15) / 16);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              if (j < nx[x]) {
                mbar_wait(&p_ready[x], n_p[x] & 1);
                ++n_p[x];
                tc_fence_after();
                attn_issue_pv(tmem_base + kAtTmemO + x * kAtD, tmem_base + x * kAtBN, ring + v_slot * kAtTile, j == 0, steps);
                if (j == nx[x] - 1) umma_commit(&o_done[x]);
              }
              if (j + 1 < nx[x]) issue_s(x, j + 1, k_slot);
            }
            umma_commit(&empty[v_slot]);
            if (j + 1 < n) umma_commit(&empty[k_slot]);
          }
        }
      }
      __syncwarp();
    } else if (warp == 2) {
      // ============================== items ==============================
      for (uint32_t k = 0;; ++k) {
        const int4 it = next;
        mbar_wait(&tab_empty[k & 1], ((k >> 1) & 1) ^ 1);
        if (lane == 0) {
          *reinterpret_cast<int4*>(smem + L::kTab + (k & 1) * 16) = it;
          mbar_arrive(&tab_full[k & 1]);
        }
        __syncwarp();
        if (it.x < 0) break;
        next = item_of(k + 1);
      }
    }
  } else {
    // ============================== softmax, epilogue ==============================
    attn_regs_softmax();
    const int x = (warp - 4) >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;                            // row of the tile == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem_base + x * kAtBN + lane_off, t_o = tmem_base + kAtTmemO + x * kAtD + lane_off;
    uint32_t n_s = 0, n_o = 0;
    for (uint32_t k = 0;; ++k) {
      const AttnItem it = attn_item(smem, tab_full, k);
      __syncwarp();
      if (lane == 0) mbar_arrive(&tab_empty[k & 1]);
      if (it.head < 0) break;
      const int n = it.blocks(x), row0 = it.q0 + x * 128, row = row0 + r;
      if (n == 0) continue;
      float m_run = -INFINITY, l_run = 0.f;
      for (int j = 0; j < n; ++j) {
        mbar_wait(&s_full[x], n_s & 1);
        ++n_s;
        tc_fence_after();
        uint32_t sv[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_s + c * 32, sv[c]);
        tmem_ld_wait();
        const int key0 = j * kAtBN;
        // only the block on the diagonal needs a mask: the others end before the tile's first row
        if (j == n - 1) attn_mask_block(sv, 0, min(row, it.len - 1) - key0, 0);
        attn_softmax_block<false>(sv, p.scale_log2, t_s, t_o, j == 0, m_run, l_run, it.len - key0 <= 64);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[x]);
      }
      // ---- O / l -> bf16, LSE ----
      mbar_wait(&o_done[x], n_o & 1);
      ++n_o;
      tc_fence_after();
      const float inv = 1.f / l_run;                           // every row sees its own key; 0 or NaN only from non-finite scores
      const bool row_ok = row < it.len;
      const long t = it.start + row;
      __nv_bfloat16* orow = p.out + t * p.o_stride_t + it.head * kAtD;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t ov[32];
        tmem_ld_32x32b_x32(t_o + c * 32, ov);
        tmem_ld_wait();
        if (!row_ok) continue;
#pragma unroll
        for (int i = 0; i < 16; ++i) ov[i] = pack_bf16x2(__uint_as_float(ov[2 * i]) * inv, __uint_as_float(ov[2 * i + 1]) * inv);
        stg_v8(orow + c * 32, ov);
        stg_v8(orow + c * 32 + 16, ov + 8);
      }
      if (row_ok && p.lse != nullptr)
        p.lse[static_cast<long>(it.head) * p.total_tokens + t] = (m_run + log2f(l_run)) * 0.6931471805599453f;
      tc_fence_before();                                       // the next item's first P V follows this thread's next p_ready
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace nrl

extern "C" cudaError_t nrl_attn_fwd_tc(const CUtensorMap* tmQ, const CUtensorMap* tmK, const CUtensorMap* tmV, void* out,
                                       float* lse, long o_stride_t, const int* cu, int num_seqs, int total, int Hq, int Hkv,
                                       float scale, int num_sms, cudaStream_t s) {
  using namespace nrl;
  if (total == 0) return cudaSuccess;
  AttnTcParams p;
  p.cu_seqlens = cu; p.out = static_cast<__nv_bfloat16*>(out); p.lse = lse; p.o_stride_t = o_stride_t;
  p.num_seqs = num_seqs; p.total_tokens = total; p.Hq = Hq; p.G = Hq / Hkv;
  p.scale_log2 = scale * 1.4426950408889634f;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnTcSmem::kTotal);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  const long most = static_cast<long>(total / kTcBM + num_seqs) * Hq;
  launch_dependent(attn_fwd_tc_kernel, static_cast<int>(most < num_sms ? most : num_sms), kAtThreads, AttnTcSmem::kTotal, s, *tmQ, *tmK, *tmV, p);
  return cudaGetLastError();
}
