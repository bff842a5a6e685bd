// Sliding-window (or chunked, or causal) attention of prompt portions on tcgen05 / TMEM / TMA, reading the 16-token bf16 pages in place:
// head size 128, the terms of NrlAttnMods except per-head score multipliers, distance slopes and distance biases
// (attention_window_mma.cu keeps those and the other head sizes).
//
// Work item: two tiles (A, B) of 128 query rows that share one key/value head -- QT consecutive tokens x HB query heads each -- which
// walk the keys their rows can see in blocks of 128 (eight pages).  One persistent CTA per SM takes every gridDim-th item,
// key heads varying fastest: 16 x 2048 tokens, 16 heads over 4, window 1024: 363 to 368 us.  The row's maximum is exact in every block (attention_tc.cuh); the other
// figures here were taken with one that could be stale by 2^8, 331 to 344 us for the same: tokens varying fastest 334 us (422 -> 624 us with 16 key
// heads and no window: the same few tiles of every sequence fell to the same CTAs); items handed out by a counter 365 us.
//   warp 0       producer: eight lanes each bring one page (two 64-column panels) of K or V by TMA into a ring of four 32 KB tiles,
//                in the order the MMAs use them (K_0, V_0, K_1, V_1, K_2 ...); keys behind the end of a sequence are zero (missing pages by an
//                out-of-range row coordinate, rows of the last page by hand), whatever a page held before
//   warp 1       MMA issuer: S_X = Q_X K^T, then per block O_X += P_X V and at once the next S_X, tiles alternating, so that the tensor
//                pipe works on one tile while the other is in its softmax
//   warp 2       finds the next item's runs (tokens of one entry) while the current one is computed; warp 3 prefetches its queries to L2
//   warps 4..11  one thread per row: scores from TMEM, cap, mask, online softmax in float with the exact maximum, O rescaled where it moved, P back
//                into TMEM over its scores; behind the last block the next item's queries (float -> bf16, swizzled), so that its first
//                scores are formed during the epilogue: sink, gate, store
// Tokens of different sequences that fall into one item are walked one run after the other over the same accumulators.
// TMEM 512 columns and 197 KB of shared memory: one CTA per SM.  Tensor pipe and 2^x on the special-function unit need 1024 clocks each per
// 128 x 128 x 128 block and tile (16 per clock and SM against 4096 multiply-adds) and neither is saturated: the hand-over between them bounds
// the walk (attention_tc.cuh); 1.0 PFLOP/s at 4 x 8192 causal tokens.  At 16 x 2048 tokens with window 1024 the query fetch and the epilogue between items cost about a third.
// Compiled WITHOUT fast-math.
#include <algorithm>

#include "attention_tc.cuh"
#include "hybrid_kernels.h"

namespace nrl {
namespace {

constexpr int kMaxTok = 256;                 // tokens per item at most (two tiles of 128 rows, one head)
constexpr int kWinSlots = 4;                 // ring of K and V tiles

struct WinTcSmem {
  static constexpr int kQ = 0;                                    // 2 tiles
  static constexpr int kRing = 2 * kAtTile;                       // kWinSlots tiles
  static constexpr int kBar = kRing + kWinSlots * kAtTile;        // mbarriers, TMEM pointer
  static constexpr int kTab = kBar + 256;                         // two run tables
  static constexpr int kTabE = 16;                                // in a table: run count, item (-1: none left) | int [kMaxTok] entry of a run
  static constexpr int kTabPos = kTabE + 4 * kMaxTok;             // int [kMaxTok]: position of its first token
  static constexpr int kTabTok = kTabPos + 4 * kMaxTok;           // uint16 [kMaxTok + 1]: its first token within the item
  static constexpr int kTabBytes = kTabTok + 2 * (kMaxTok + 8);
  static constexpr int kTotal = kTab + 2 * kTabBytes;
};
static_assert(WinTcSmem::kTotal <= 227 * 1024 && WinTcSmem::kTabBytes % 16 == 0, "shared memory of one CTA");

struct WinTcParams {
  const float* q;
  long sq;
  const int* block_table;
  int max_blocks;
  const int* tok_entry;
  const int* pos;
  int window;
  float scale, out_scale;
  __nv_bfloat16* out;
  long so;
  int T, Hq, Hkv, HB, QT, oob_k, oob_v;      // oob: a row coordinate behind the page pool (TMA fills zeros)
  int ntiles, nitems;
  NrlAttnMods md;
};

__device__ __forceinline__ int first_key(int p, int window, int chunked) { return chunked ? p - p % window : p - window + 1; }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
// cap * tanh(x / cap), tanh(z) = (1 - e) / (1 + e) with e = exp(-2 |z|)
__device__ __forceinline__ float softcap_f(float x, float cap, float inv_cap) {
  const float e = ex2_approx(-2.885390081777927f * fabsf(x * inv_cap));
  return copysignf(cap * __fdividef(1.f - e, 1.f + e), x);
}

struct Item {
  int g, h0, hb, t_begin, ntok;
  __device__ __forceinline__ Item(const WinTcParams& p, int item) {
    const int per_g = p.Hq / p.Hkv, heads = p.nitems / p.ntiles, x = item / heads, gz = item - x * heads, z = gz / p.Hkv;
    g = gz - z * p.Hkv;
    h0 = g * per_g + z * p.HB;
    hb = min(p.HB, per_g - z * p.HB);
    t_begin = (p.ntiles - 1 - x) * 2 * p.QT;                 // late tokens see more keys: they start first
    ntok = min(p.T - t_begin, 2 * p.QT);
  }
};

// The key blocks of an item in the order all roles walk them: run after run, kept first keys in front of the window's blocks.
struct Walk {
  const int *run_e, *run_pos;
  const uint16_t* run_tok;
  int nruns, QT, window, chunked, keep;
  int r, ib, nblk, nkb, kb0, hi, t0, t1, p0;
  int vlo0, vhi0, vlo1, vhi1;                                        // keys the tiles' rows of this run see (last -1: none)
  __device__ __forceinline__ void visible(int a, int b, int& lo, int& last) const {
    lo = a <= b ? first_key(p0 + a - t0, window, chunked) : 0;
    last = a <= b ? p0 + b - t0 : -1;
  }
  __device__ __forceinline__ void load_run() {
    t0 = run_tok[r];
    t1 = run_tok[r + 1];
    p0 = run_pos[r];
    hi = p0 + (t1 - t0) - 1;
    kb0 = max(0, first_key(p0, window, chunked)) & ~(kAtBN - 1);
    nkb = keep > 0 ? (min(keep, kb0) + kAtBN - 1) / kAtBN : 0;
    nblk = nkb + (hi - kb0) / kAtBN + 1;
    ib = 0;
    visible(t0, min(t1, QT) - 1, vlo0, vhi0);
    visible(max(t0, QT), t1 - 1, vlo1, vhi1);
  }
  __device__ __forceinline__ void init(const WinTcParams& p, const uint8_t* tab) {
    run_e = reinterpret_cast<const int*>(tab + WinTcSmem::kTabE);
    run_pos = reinterpret_cast<const int*>(tab + WinTcSmem::kTabPos);
    run_tok = reinterpret_cast<const uint16_t*>(tab + WinTcSmem::kTabTok);
    nruns = *reinterpret_cast<const int*>(tab);
    QT = p.QT; window = p.window; chunked = p.md.chunked;
    keep = p.md.chunked ? 0 : p.md.keep_first;
    r = 0;
    load_run();
  }
  __device__ __forceinline__ bool live() const { return r < nruns; }
  __device__ __forceinline__ void next() {
    if (++ib == nblk && ++r < nruns) load_run();
  }
  __device__ __forceinline__ int kb() const { return ib < nkb ? ib * kAtBN : kb0 + (ib - nkb) * kAtBN; }
  __device__ __forceinline__ bool part(int x) const {               // does tile x see a key of this block
    const int k = kb();
    return k <= (x == 0 ? vhi0 : vhi1) && (k + kAtBN - 1 >= (x == 0 ? vlo0 : vlo1) || k < keep);
  }
};

// the item of table `k` (waits for the table); -1: none left
__device__ __forceinline__ int next_item(const uint8_t* smem, uint64_t* tab_full, uint32_t k) {
  mbar_wait(&tab_full[k & 1], (k >> 1) & 1);
  return reinterpret_cast<const volatile int*>(smem + WinTcSmem::kTab + (k & 1) * WinTcSmem::kTabBytes)[1];
}

// Queries of one tile (float -> bf16, swizzled): a warp converts 32 rows, two rows per load (16 lanes x 8 columns each), all in flight.
__device__ __forceinline__ void load_queries(const WinTcParams& p, const Item& it, int x, int w4, int lane, uint8_t* tile) {
  const int r0 = w4 * 32 + (lane >> 4), c16 = lane & 15;
  const float* base = p.q + static_cast<long>(it.t_begin) * p.sq + static_cast<long>(it.h0) * kAtD + c16 * 8;
  int tt = x * p.QT + r0 / p.HB, hh = r0 % p.HB;
  float f[16][8];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (r0 + 2 * i < p.QT * p.HB && tt < it.ntok && hh < it.hb) {
      ldg_v8(base + static_cast<long>(tt) * p.sq + hh * kAtD, f[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[i][j] = 0.f;
    }
    hh += 2;
    if (hh >= p.HB) { hh -= p.HB; ++tt; }
    if (hh >= p.HB) { hh -= p.HB; ++tt; }                      // one head per row group: two tokens on
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = r0 + 2 * i;
    uint8_t* dst = tile + (c16 >> 3) * kAtPanel + r * 128 + (((c16 & 7) ^ (r & 7)) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(f[i][0], f[i][1]), pack_bf16x2(f[i][2], f[i][3]), pack_bf16x2(f[i][4], f[i][5]),
                                                pack_bf16x2(f[i][6], f[i][7]));
  }
  fence_proxy_async_smem();
}

__global__ void __launch_bounds__(kAtThreads, 1)
window_attention_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const WinTcParams p) {
  using L = WinTcSmem;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBar);      // [kWinSlots]
  uint64_t* empty = full + kWinSlots;          // [kWinSlots]
  uint64_t* q_full = empty + kWinSlots;        // [tile]
  uint64_t* s_full = q_full + 2;               // [tile]
  uint64_t* p_ready = s_full + 2;              // [tile]
  uint64_t* o_done = p_ready + 2;              // [tile]
  uint64_t* tab_full = o_done + 2;             // [2]
  uint64_t* tab_empty = tab_full + 2;          // [2]
  uint64_t* tail_bar = tab_empty + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tail_bar + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int i = 0; i < kWinSlots; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&empty[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&q_full[i], 4);
        mbar_init(&s_full[i], 1);
        mbar_init(&p_ready[i], 4);
        mbar_init(&o_done[i], 1);
        mbar_init(&tab_full[i], 1);
        mbar_init(&tab_empty[i], 11);          // producer, MMA issuer, prefetcher, eight softmax warps
      }
      mbar_init(tail_bar, 1);
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_ptr, 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  if (warp < 4) {
    attn_regs_issue();
    if (warp == 0) {
      // ============================== producer ==============================
      int slot = 0;
      uint32_t phase = 0, tail_phase = 0;
      for (uint32_t k = 0;; ++k) {
        const int item = next_item(smem, tab_full, k);
        if (item < 0) break;
        const Item it(p, item);
        const int gv = p.md.v_div > 1 ? it.g / p.md.v_div : it.g, Hv = p.md.v_div > 1 ? p.Hkv / p.md.v_div : p.Hkv;
        Walk wk;
        for (wk.init(p, smem + L::kTab + (k & 1) * L::kTabBytes); wk.live(); wk.next()) {
          const int kb = wk.kb(), hi = wk.hi;
          const int* bt = p.block_table + static_cast<long>(wk.run_e[wk.r]) * p.max_blocks;
          int page = -1;                                            // lane l: page l of the block
          if (lane < 8 && kb + 16 * lane <= hi) page = bt[(kb >> 4) + lane];
#pragma unroll
          for (int kv = 0; kv < 2; ++kv) {
            mbar_wait(&empty[slot], phase ^ 1);
            uint8_t* dst = smem + L::kRing + slot * kAtTile;
            const bool tail = kv == 1 && hi < kb + kAtBN - 1 && ((hi + 1) & 15) != 0;      // V rows behind the sequence's end inside a page
            uint64_t* bar = tail ? tail_bar : &full[slot];
            if (lane == 0) mbar_arrive_expect_tx(bar, kAtTile);
            __syncwarp();
            if (lane < 8) {
              const int heads = kv == 0 ? p.Hkv : Hv, head = kv == 0 ? it.g : gv;
              const int row = page < 0 ? (kv == 0 ? p.oob_k : p.oob_v) : (page * heads + head) * 16;
              const CUtensorMap* tm = kv == 0 ? &tmK : &tmV;
              tma_load_2d(dst + lane * 2048, tm, bar, 0, row);
              tma_load_2d(dst + kAtPanel + lane * 2048, tm, bar, 64, row);
            }
            __syncwarp();
            if (tail) {
              mbar_wait(tail_bar, tail_phase);
              tail_phase ^= 1;
              const int from = (hi - kb) + 1, to = (from + 15) & ~15;                    // rows [from, to) of the last page
              for (int i = lane; i < (to - from) * 16; i += 32) {
                const int row = from + (i >> 4), c = i & 15;
                *reinterpret_cast<uint4*>(dst + (c >> 3) * kAtPanel + row * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
              }
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) mbar_arrive(&full[slot]);
            }
            if (++slot == kWinSlots) { slot = 0; phase ^= 1; }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&tab_empty[k & 1]);
      }
    } else if (warp == 1) {
      // ============================== MMA issuer ==============================
      if (elect_one()) {
        int slot = 0;                            // ring slot of the next tile in load order
        uint32_t phase = 0, n_p[2] = {0, 0}, n_q[2] = {0, 0};
        auto ring_next = [&]() {
          if (++slot == kWinSlots) { slot = 0; phase ^= 1; }
        };
        const uint32_t q_addr = smem_u32(smem + L::kQ), ring = smem_u32(smem + L::kRing);
        for (uint32_t k = 0; next_item(smem, tab_full, k) >= 0; ++k) {
          Walk wk;
          wk.init(p, smem + L::kTab + (k & 1) * L::kTabBytes);
          bool fresh[2] = {true, true}, first[2] = {true, true};    // no scores / no P V of this item issued yet
          auto issue_s = [&](int x, int s) {
            if (fresh[x]) {
              mbar_wait(&q_full[x], n_q[x] & 1);
              ++n_q[x];
              tc_fence_after();
              fresh[x] = false;
            }
            attn_issue_s(tmem_base + x * kAtBN, q_addr + x * kAtTile, ring + s * kAtTile);
            umma_commit(&s_full[x]);
          };
          mbar_wait(&full[slot], phase);
          tc_fence_after();
#pragma unroll
          for (int x = 0; x < 2; ++x)
            if (wk.part(x)) issue_s(x, slot);
          umma_commit(&empty[slot]);
          ring_next();
          while (wk.live()) {
            const bool pv[2] = {wk.part(0), wk.part(1)};
            bool more[2] = {false, false};
            wk.next();
            const bool has_next = wk.live();
            if (has_next) {
              more[0] = wk.part(0);
              more[1] = wk.part(1);
            }
            // load order is K_0, V_0, K_1, V_1, K_2 ...: V of this block sits in `slot`, K of the next one behind it
            const int v_slot = slot;
            mbar_wait(&full[v_slot], phase);
            ring_next();
            const int k_slot = slot;
            if (has_next) {
              mbar_wait(&full[k_slot], phase);
              ring_next();
            }
            tc_fence_after();
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              if (pv[x]) {
                mbar_wait(&p_ready[x], n_p[x] & 1);
                ++n_p[x];
                tc_fence_after();
                attn_issue_pv(tmem_base + kAtTmemO + x * kAtD, tmem_base + x * kAtBN, ring + v_slot * kAtTile, first[x]);
                first[x] = false;
              }
              if (more[x]) issue_s(x, k_slot);
            }
            umma_commit(&empty[v_slot]);
            if (has_next) umma_commit(&empty[k_slot]);
          }
#pragma unroll
          for (int x = 0; x < 2; ++x)
            if (!first[x]) umma_commit(&o_done[x]);
          mbar_arrive(&tab_empty[k & 1]);
        }
      }
      __syncwarp();
    } else if (warp == 2) {
      // ============================== run tables ==============================
      int item = blockIdx.x;
      for (uint32_t k = 0;; ++k, item += gridDim.x) {
        mbar_wait(&tab_empty[k & 1], ((k >> 1) & 1) ^ 1);
        uint8_t* tab = smem + L::kTab + (k & 1) * L::kTabBytes;
        if (item >= p.nitems) {
          if (lane == 0) {
            reinterpret_cast<int*>(tab)[1] = -1;
            mbar_arrive(&tab_full[k & 1]);
          }
          break;
        }
        const Item it(p, item);
        int* run_e = reinterpret_cast<int*>(tab + L::kTabE);
        int* run_pos = reinterpret_cast<int*>(tab + L::kTabPos);
        uint16_t* run_tok = reinterpret_cast<uint16_t*>(tab + L::kTabTok);
        int e[kMaxTok / 32], before[kMaxTok / 32], ps[kMaxTok / 32];
#pragma unroll
        for (int i = 0; i < kMaxTok / 32; ++i) {
          const int t = i * 32 + lane;
          e[i] = t < it.ntok ? p.tok_entry[it.t_begin + t] : -1;
          before[i] = t < it.ntok && t > 0 ? p.tok_entry[it.t_begin + t - 1] : -1;
          ps[i] = t < it.ntok ? p.pos[it.t_begin + t] : 0;
        }
        int n = 0;
#pragma unroll
        for (int i = 0; i < kMaxTok / 32; ++i) {
          const int t = i * 32 + lane;
          const bool begins = t < it.ntok && (t == 0 || e[i] != before[i]);
          const uint32_t m = __ballot_sync(0xffffffffu, begins);
          if (begins) {
            const int at = n + __popc(m & ((1u << lane) - 1));
            run_e[at] = e[i];
            run_pos[at] = ps[i];
            run_tok[at] = static_cast<uint16_t>(t);
          }
          n += __popc(m);
        }
        if (lane == 0) {
          run_tok[n] = static_cast<uint16_t>(it.ntok);
          reinterpret_cast<int*>(tab)[0] = n;
          reinterpret_cast<int*>(tab)[1] = item;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&tab_full[k & 1]);
      }
    } else {
      // ============================== L2 prefetch of the next item's queries ==============================
      for (uint32_t k = 0;; ++k) {
        const int item = next_item(smem, tab_full, k);
        if (item < 0) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(&tab_empty[k & 1]);
        if (k == 0) continue;                                      // the first item's queries are being loaded already
        const Item it(p, item);
        const int lines = it.hb * 4;                               // 128-byte lines per token
        for (int i = lane; i < it.ntok * lines; i += 32) {
          const int tt = i / lines, c = i - tt * lines;
          const float* a = p.q + static_cast<long>(it.t_begin + tt) * p.sq + static_cast<long>(it.h0) * kAtD + c * 32;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
        }
      }
    }
  } else {
    // ============================== softmax, next queries, epilogue ==============================
    attn_regs_softmax();
    const int x = (warp - 4) >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;                            // row of the tile == TMEM lane
    const int trel = x * p.QT + r / p.HB, hh = r % p.HB;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem_base + x * kAtBN + lane_off, t_o = tmem_base + kAtTmemO + x * kAtD + lane_off;
    const bool capped = p.md.softcap > 0.f;
    const float inv_cap = capped ? 1.f / p.md.softcap : 0.f;
    const float sl2 = capped ? 1.4426950408889634f : p.scale * 1.4426950408889634f;
    uint32_t n_s = 0, n_o = 0;
    auto fetch = [&](int item) {
      const Item it(p, item);
      if (x * p.QT >= it.ntok) return;
      load_queries(p, it, x, quad, lane, smem + L::kQ + x * kAtTile);
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full[x]);
    };
    int item = blockIdx.x, next = 0;
    fetch(item);
    for (uint32_t k = 0; item >= 0; ++k, item = next) {
      float m_run = -INFINITY, l_run = 0.f;
      bool any = false;
      {
        const Item it(p, item);
        const bool row_ok = r < p.QT * p.HB && trel < it.ntok && hh < it.hb;
        const int tile_t0 = x * p.QT, tile_t1 = min((x + 1) * p.QT, it.ntok);
        mbar_wait(&tab_full[k & 1], (k >> 1) & 1);
        Walk wk;
        for (wk.init(p, smem + L::kTab + (k & 1) * L::kTabBytes); wk.live(); wk.next()) {
          if (!wk.part(x)) continue;
          const int kb = wk.kb();
          mbar_wait(&s_full[x], n_s & 1);
          ++n_s;
          tc_fence_after();
          uint32_t sv[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_s + c * 32, sv[c]);
          tmem_ld_wait();
          if (capped) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i) sv[c][i] = __float_as_uint(softcap_f(__uint_as_float(sv[c][i]) * p.scale, p.md.softcap, inv_cap));
          }
          // a block that every row of the tile sees whole needs no mask (rows without a query may compute what they like)
          const bool interior = wk.t0 <= tile_t0 && wk.t1 >= tile_t1 && kb + kAtBN - 1 <= wk.p0 + (tile_t0 - wk.t0) &&
                                kb >= first_key(wk.p0 + (tile_t1 - 1 - wk.t0), wk.window, wk.chunked);
          if (!interior) {
            const bool act = row_ok && trel >= wk.t0 && trel < wk.t1;
            const int pq = act ? wk.p0 + (trel - wk.t0) - kb : -1;           // last and first visible key, relative to the block
            const int plo = first_key(wk.p0 + (trel - wk.t0), wk.window, wk.chunked) - kb;
            attn_mask_block(sv, plo, pq, wk.keep - kb);
          }
          attn_softmax_block<true>(sv, sl2, t_s, t_o, !any, m_run, l_run);
          any = true;
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_ready[x]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&tab_empty[k & 1]);
      }
      // every score product of this tile has retired (its last result was read above): its query buffer is free
      next = next_item(smem, tab_full, k + 1);
      if (next >= 0) fetch(next);
      if (!any) continue;
      // ---- out = out_scale * O / l ----
      mbar_wait(&o_done[x], n_o & 1);
      ++n_o;
      tc_fence_after();
      const Item it(p, item);
      const bool row_ok = r < p.QT * p.HB && trel < it.ntok && hh < it.hb;
      const int h = it.h0 + hh;
      const long t = it.t_begin + trel;
      float f = l_run > 0.f ? p.out_scale / l_run : 0.f;
      if (l_run != l_run) f = l_run;                           // a row whose scores hold NaN stays NaN
      if (row_ok && p.md.head_sink != nullptr) {               // one more term in the denominator: a score with no key and no value
        const float s2 = p.md.head_sink[h] * 1.4426950408889634f, mt = fmaxf(m_run, s2), fo = ex2_approx(m_run - mt);
        f = p.out_scale * fo / (l_run * fo + ex2_approx(s2 - mt));
      }
      const float* gcol = nullptr;                             // one gate per output column
      if (row_ok && p.md.gate != nullptr) {
        if (p.md.gate_cols) gcol = p.md.gate + t * p.md.gate_stride + static_cast<long>(h) * kAtD;
        else f *= sigmoid_f(p.md.gate[t * p.md.gate_stride + h]);
      }
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t ov[32];
        tmem_ld_32x32b_x32(t_o + c * 32, ov);
        tmem_ld_wait();
        if (!row_ok) continue;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float v = __uint_as_float(ov[i]) * f;
          if (gcol != nullptr) v *= sigmoid_f(gcol[c * 32 + i]);
          ov[i] = __float_as_uint(v);
        }
        if (p.md.out_float != nullptr) {
          float* dst = p.md.out_float + t * p.md.out_float_stride + static_cast<long>(h) * kAtD + c * 32;
#pragma unroll
          for (int i = 0; i < 32; i += 8) stg_v8(dst + i, ov + i);
        } else {
          __nv_bfloat16* dst = p.out + t * p.so + static_cast<long>(h) * kAtD + c * 32;
#pragma unroll
          for (int i = 0; i < 16; ++i) ov[i] = pack_bf16x2(__uint_as_float(ov[2 * i]), __uint_as_float(ov[2 * i + 1]));
          stg_v8(dst, ov);
          stg_v8(dst + 16, ov + 8);
        }
      }
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

}  // namespace
}  // namespace nrl

extern "C" {

int nrl_window_attention_tc_fits(const float* q, long sq, const void* out, long so, long T, int Hq, int Hkv, int D, int Dv, int page, float scale,
                                 const NrlAttnMods* md) {
  if (page != 16 || D != nrl::kAtD || Dv != nrl::kAtD || Hkv < 1 || Hq % Hkv != 0 || Hq / Hkv > 128 || !(scale > 0.f)) return 0;
  if (md->head_scale != nullptr || md->head_slope != nullptr || md->dist_bias != nullptr || md->kv_shared || md->q_head_stride != 0) return 0;
  // 32-byte accesses to the queries and the result
  if (reinterpret_cast<uintptr_t>(q) % 32 != 0 || sq % 8 != 0) return 0;
  if (md->out_float != nullptr) {
    if (reinterpret_cast<uintptr_t>(md->out_float) % 32 != 0 || md->out_float_stride % 8 != 0) return 0;
  } else if (reinterpret_cast<uintptr_t>(out) % 32 != 0 || so % 16 != 0) {
    return 0;
  }
  return T >= 1 && T < (1L << 24);
}

// Tokens of a tile.  An item walks its runs one after the other, so a step of many short portions in few items waits for a few CTAs.  There the tiles
// take as few tokens as give every SM an item (in brackets: full tiles, mma.sync form): 64 portions of 4 tokens, 16 heads over 16, 35 us (155, 100), behind
// 1000 keys 159 (1098, 1421); 16 over 4, 20 (49, 34); 200 single tokens behind 1000 keys beside a portion of 30, 16 over 16, 474 (3396, 5633).
// Not where the portions are long: an item that holds one whole portion has one run, a smaller one that lies across two has two (16 portions of
// 64 behind 1000 keys, 16 over 4: 32 us, with small tiles 57).
int nrl_window_attention_tc_tokens(long T, long E, int Hq, int Hkv, int num_sms) {
  const int per_g = Hq / Hkv, HB = per_g < 128 ? per_g : 128, most = 128 / HB;
  const int heads = Hkv * ((per_g + HB - 1) / HB), share = num_sms / heads;          // items of one stretch of tokens; stretches that the SMs hold
  if (share < 1 || E < 1) return most;
  const long qt = (T + 2 * share - 1) / (2 * share);
  const long runs_T = std::min(E * T, 2 * most * E);                                 // runs of a full item, times T: E, or its tokens by the mean portion
  return qt < most && runs_T > T + 2 * qt * E ? static_cast<int>(qt) : most;
}

cudaError_t nrl_window_attention_tc(const CUtensorMap* tmK, const CUtensorMap* tmV, int oob_k, int oob_v, const float* q, long sq,
                                    const int* block_table, int max_blocks, const int* tok_entry, const int* pos, int window, float scale,
                                    float out_scale, void* out, long so, int T, int E, int Hq, int Hkv, const NrlAttnMods* md, int num_sms,
                                    cudaStream_t s) {
  using namespace nrl;
  if (T <= 0) return cudaSuccess;
  if (window < 1 || Hkv < 1 || Hq % Hkv != 0 || (md->v_div > 1 && Hkv % md->v_div != 0)) return cudaErrorInvalidValue;
  WinTcParams p;
  p.q = q; p.sq = sq; p.block_table = block_table; p.max_blocks = max_blocks; p.tok_entry = tok_entry; p.pos = pos; p.window = window;
  p.scale = scale; p.out_scale = out_scale; p.out = static_cast<__nv_bfloat16*>(out); p.so = so; p.T = T; p.Hq = Hq; p.Hkv = Hkv;
  const int per_g = Hq / Hkv;
  p.HB = per_g < 128 ? per_g : 128;
  p.QT = nrl_window_attention_tc_tokens(T, E, Hq, Hkv, num_sms);
  p.oob_k = oob_k; p.oob_v = oob_v; p.md = *md;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(window_attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WinTcSmem::kTotal);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  p.ntiles = (T + 2 * p.QT - 1) / (2 * p.QT);
  p.nitems = p.ntiles * Hkv * ((per_g + p.HB - 1) / p.HB);
  window_attention_tc_kernel<<<p.nitems < num_sms ? p.nitems : num_sms, kAtThreads, WinTcSmem::kTotal, s>>>(*tmK, *tmV, p);
  return cudaGetLastError();
}

}  // extern "C"
