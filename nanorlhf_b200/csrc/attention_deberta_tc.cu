// DeBERTa disentangled attention (not causal, packed varlen, head size 64) on tcgen05 / TMEM / TMA for sm_100a:
//   score(i, j) = (q_i . k_j + A[i, c] + B[j, c]) * scale,  c = bucket of i - j,  A = Q Kr^T (content to position), B = K Qr^T (position to content)
//
// Work item: 128 query rows of one head.  A's rows are formed here, 64 buckets at a time as score tiles of Q against the position keys, rounded to bf16 as
// a GEMM would leave them, and stay in shared memory for the whole walk over the keys; B comes from global memory, for every block of 64 keys the
// columns that its scores can meet.  Two softmax warpgroups take the score tiles in turn, each with its own maximum, sum and O; they are merged at the end.
//   warp 0        position keys, K and V tiles
//   warp 1        scores, up to four tiles ahead of the softmax, across items too
//   warp 2        P V
//   warp 3        finds the next item
//   warps 4..19   a row and half of the columns each: A tiles into shared memory; then scores + A + B, online softmax, P as bf16 into TMEM over the scores
//   warps 20..23  the next item's queries into TMEM; three of them a block of keys each in turn: the buckets of its 191 differences and B's columns (per 8 keys 144 of
//                 them: 135 differences and the alignment)
// A block whose differences all fall into one bucket (from 511 positions on) needs no lookup: A is a number per row and B one per key.
// One persistent CTA per SM; items go from the longest to the shortest sequence, dealt to the CTAs forwards and backwards in turn.
//
// What bounds it: the chain of one tile, above all its lookups (two and a half reads of shared memory a score; without them it took 0.69 of its time, without
// P V and 2^x too 0.55).  The streams take turns at them (2 %); all loads in front of the first sum, sums of A and B before the scores are there and longer
// sleeps of the waiting warps changed nothing or cost up to 8 %.  The maximum is the row's own in every block, which both halves of a row agree on through tensor
// memory: 16 x 1536 tokens with 16 heads 524 us in a graph, 486 with one that may be stale by 2^8, whose error against float64 was up to 1.21 times that of the
// mma.sync form (operands of standard deviation 1.5; now 0.98); asking first whether any row moved 562.
// The mma.sync form with both tables in global memory takes 767 us and 90 more for the second table, and is bound by the windows that it fetches (5 GB through
// the L2, 1.1 here): 16 x 300 tokens 55 against 54 + 23, 4 x 700 49 / 59 + 14, 16 x 40 10.7 / 6.7 + 7.9, so that it is left only where A does not fit (more than 512
// buckets).
#include "attention_tc.cuh"
#include "kernels.h"
#include "launch.h"

namespace nrl {
namespace {

constexpr int kDbThreads = 768;            // registers: 768 x 80 at launch = 128 x (56 + 4 x 88 + 72)
constexpr int kDbBM = 128, kDbBN = 64;     // query rows per item, keys per block
constexpr int kDbTile = 64 * 128;          // [64 rows][64 x bf16], 128B-swizzled
constexpr int kDbWin = 144;                // columns of B staged per 8 keys
constexpr int kDbStages = 3;
constexpr int kDbAPitch = 1028;            // bytes: 512 buckets; 257 words, so that rows lie one bank apart
constexpr int kDbMaxBuckets = 512;

struct DbSmem {
  static constexpr int kK = 0;                                   // two tiles
  static constexpr int kV = kK + 2 * kDbTile;                    // kDbStages tiles
  static constexpr int kB = kV + kDbStages * kDbTile;            // per stage: B | buckets (two copies, one shifted by an entry) | per 8 keys where column 0 lies, flag
  static constexpr int kLut = kDbBN * kDbWin * 2;
  static constexpr int kLutCopy = 448;                           // 192 entries, and the copies 16 banks apart
  static constexpr int kMeta = kLut + 2 * kLutCopy;
  static constexpr int kStage = kMeta + 128;                     // a multiple of 128
  static constexpr int kA = kB + kDbStages * kStage;
  static constexpr int kBar = kA + kDbBM * kDbAPitch;
  static constexpr int kTab = kBar + 320;                        // two items of 8 ints
  static constexpr int kTotal = kTab + 2 * 32;
};
static_assert(DbSmem::kStage % 128 == 0 && DbSmem::kBar % 16 == 0 && DbSmem::kTotal <= 227 * 1024, "shared memory");

// TMEM columns: scores [stream][2] (P over the first 32 of them) | O [stream] | Q [2] | maximum and sum | maxima of a tile
constexpr int kDbTmemO = 256, kDbTmemQ = 384, kDbTmemML = 448, kDbTmemMax = 456;      // ... | [stream][half] | [stream][tile & 1][half]

struct DbParams {
  const int* cu_seqlens;
  const __nv_bfloat16* q;
  __nv_bfloat16* out;
  const short* lut;           // entry lut_center + i - j
  long q_stride_t, o_stride_t;
  int num_seqs, total_tokens, heads, lut_center, buckets;
  float scale_log2;
  NRL_DEVICE int bucket(int diff) const {
    return min(max(static_cast<int>(__ldg(lut + lut_center + min(max(diff, -lut_center), lut_center))), 0), buckets - 1);
  }
};

// Warps that wait for long sleep between tries: every try takes a slot of the pipe that the lookups go through.
template <int NS>
NRL_DEVICE void db_wait_idle(uint64_t* bar, uint32_t parity) {
  for (uint32_t n = 0; !mbar_try_wait(bar, parity);) {
    __nanosleep(NS);
    if (++n == (1u << 24)) __trap();
  }
}
// Stages are filled by a warp each, so a stream may come to a block before the one that its stage holds first has been filled, when the barrier's parity tells
// nothing: the number beside the buckets says whose they are.
NRL_DEVICE void db_wait_block(uint32_t addr, uint32_t number) {
  for (uint32_t n = 0;;) {
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    if (v == number) return;
    __nanosleep(20);
    if (++n == (1u << 26)) __trap();
  }
}

struct DbItem {
  int head, q0, start, len, tile0, tiles;        // A tiles (64 buckets each) tile0 .. tile0 + tiles - 1; head -1: none left
  NRL_DEVICE int blocks() const { return (len + kDbBN - 1) / kDbBN; }
};
NRL_DEVICE DbItem db_item(const uint8_t* smem, uint64_t* tab_full, uint32_t k) {
  db_wait_idle<100>(&tab_full[k & 1], (k >> 1) & 1);
  const volatile int* t = reinterpret_cast<const volatile int*>(smem + DbSmem::kTab + (k & 1) * 32);
  return {t[0], t[1], t[2], t[3], t[4], t[5]};
}

NRL_DEVICE void sts_u16(uint32_t addr, uint32_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(static_cast<unsigned short>(v)) : "memory"); }
NRL_DEVICE void sts_u32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
// f + the bf16 at a shared address
template <int OFFSET = 0>
NRL_DEVICE float add_lds_bf16(float f, uint32_t addr) {
  float r;
  asm volatile("{\n\t.reg .b16 h;\n\tld.shared.b16 h, [%2 + %3];\n\tadd.rn.f32.bf16 %0, h, %1;\n\t}" : "=f"(r) : "f"(f), "r"(addr), "n"(OFFSET));
  return r;
}
// Scores of 32 keys + A + B, two keys from column I on at a time: `lut` holds their offsets as a pair of 16 bits; a dot product with (1, 0) or (0, 1) takes one of
// them out and adds the row.
template <int I = 0>
NRL_DEVICE void db_add_tables(uint32_t (&sv)[32], uint32_t lut, uint32_t a_row, const uint32_t (&b_row)[4]) {
  if constexpr (I < 32) {
    uint32_t x;
    asm volatile("ld.shared.u32 %0, [%1 + %2];" : "=r"(x) : "r"(lut), "n"(I * 2));
    sv[I] = __float_as_uint(add_lds_bf16<I * kDbWin * 2>(add_lds_bf16(__uint_as_float(sv[I]), __dp2a_lo(x, 0x0001u, a_row)), __dp2a_lo(x, 0x0001u, b_row[I >> 3])));
    sv[I + 1] = __float_as_uint(add_lds_bf16<(I + 1) * kDbWin * 2>(add_lds_bf16(__uint_as_float(sv[I + 1]), __dp2a_lo(x, 0x0100u, a_row)), __dp2a_lo(x, 0x0100u, b_row[I >> 3])));
    db_add_tables<I + 2>(sv, lut, a_row, b_row);
  }
}
// the same where all differences fall into one bucket: a number per key, 16 bytes apart
template <int I = 0>
NRL_DEVICE void db_add_column(uint32_t (&sv)[32], uint32_t b_col) {
  if constexpr (I < 32) {
    sv[I] = __float_as_uint(add_lds_bf16<I * 16>(__uint_as_float(sv[I]), b_col));
    db_add_column<I + 1>(sv, b_col);
  }
}
NRL_DEVICE void tmem_st_x1(uint32_t taddr, uint32_t a) { asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(a) : "memory"); }
// the larger of two columns
NRL_DEVICE float tmem_max_x2(uint32_t taddr) {
  uint32_t a, b;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(taddr) : "memory");
  tmem_ld_wait();
  return fmaxf(__uint_as_float(a), __uint_as_float(b));
}
NRL_DEVICE void tmem_st_x2(uint32_t taddr, uint32_t a, uint32_t b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}

__global__ void __launch_bounds__(kDbThreads, 1)
deberta_attn_tc_kernel(const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                       const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmB1, const DbParams p) {
  using L = DbSmem;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* k_full = reinterpret_cast<uint64_t*>(smem + L::kBar);      // [2]
  uint64_t* k_empty = k_full + 2;              // [2]
  uint64_t* v_full = k_empty + 2;              // [kDbStages]
  uint64_t* v_empty = v_full + kDbStages;      // [kDbStages]
  uint64_t* b_full = v_empty + kDbStages;      // [kDbStages]
  uint64_t* b_empty = b_full + kDbStages;      // [kDbStages]
  uint64_t* s_full = b_empty + kDbStages;      // [stream * 2 + buffer]
  uint64_t* s_free = s_full + 4;               // [stream * 2 + buffer]
  uint64_t* p_ready = s_free + 4;              // [stream * 2 + buffer]
  uint64_t* pv_done = p_ready + 4;             // [stream]
  uint64_t* q_ready = pv_done + 2;             // [2]
  uint64_t* q_free = q_ready + 2;              // [2]
  uint64_t* tab_full = q_free + 2;             // [2]
  uint64_t* tab_empty = tab_full + 2;          // [2]
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tab_empty + 2);
  static_assert((2 + 2 + 4 * kDbStages + 4 + 4 + 4 + 2 + 2 + 2 + 2 + 2) * 8 + 4 <= 320, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmP);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmB1);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int i = 0; i < 2; ++i) {
        mbar_init(&k_full[i], 1);
        mbar_init(&k_empty[i], 1);
        mbar_init(&pv_done[i], 1);
        mbar_init(&q_ready[i], 4);
        mbar_init(&q_free[i], 1);
        mbar_init(&tab_full[i], 1);
        mbar_init(&tab_empty[i], 23);          // warps 0, 1, 2, sixteen softmax warps, four query warps
      }
      for (int i = 0; i < kDbStages; ++i) {
        *reinterpret_cast<int*>(smem + L::kB + i * L::kStage + L::kMeta + 36) = -1;
        mbar_init(&v_full[i], 1);
        mbar_init(&v_empty[i], 1);
        mbar_init(&b_full[i], 2);              // the copies; the buckets
        mbar_init(&b_empty[i], 8);             // the warps of a stream
      }
      for (int i = 0; i < 4; ++i) {
        mbar_init(&s_full[i], 1);
        mbar_init(&s_free[i], 1);
        mbar_init(&p_ready[i], 8);
      }
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_ptr, 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  pdl_wait();
  pdl_launch_dependents();

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
      // ============================== position keys, K and V ==============================
      if (elect_one()) {
        uint32_t f = 0, n_v = 0;                 // tiles so far; slot f & 1
        auto load = [&](const CUtensorMap* tm, int col, int row) {
          db_wait_idle<100>(&k_empty[f & 1], ((f >> 1) & 1) ^ 1);
          mbar_arrive_expect_tx(&k_full[f & 1], kDbTile);
          tma_load_2d(smem + L::kK + (f & 1) * kDbTile, tm, &k_full[f & 1], col, row);
          ++f;
        };
        for (uint32_t k = 0;; ++k) {
          const DbItem it = db_item(smem, tab_full, k);
          mbar_arrive(&tab_empty[k & 1]);
          if (it.head < 0) break;
          for (int t = 0; t < it.tiles; ++t) load(&tmP, it.head * 64, (it.tile0 + t) * 64);
          for (int j = 0; j < it.blocks(); ++j, ++n_v) {
            load(&tmK, it.head * 64, it.start + j * kDbBN);
            const uint32_t s = n_v % kDbStages;
            db_wait_idle<100>(&v_empty[s], ((n_v / kDbStages) & 1) ^ 1);
            mbar_arrive_expect_tx(&v_full[s], kDbTile);
            tma_load_2d(smem + L::kV + s * kDbTile, &tmV, &v_full[s], it.head * 64, it.start + j * kDbBN);
          }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ============================== scores ==============================
      // tile f of all items goes to stream f & 1, buffer (f >> 1) & 1
      if (elect_one()) {
        constexpr uint32_t idesc = make_idesc(128, 64, 1, 1);
        uint32_t f = 0;
        for (uint32_t k = 0;; ++k) {
          const DbItem it = db_item(smem, tab_full, k);
          mbar_arrive(&tab_empty[k & 1]);
          if (it.head < 0) break;
          mbar_wait_quiet(&q_ready[k & 1], (k >> 1) & 1);
          const uint32_t t_q = tmem_base + kDbTmemQ + (k & 1) * 32;
          for (int t = it.tiles + it.blocks(); t > 0; --t, ++f) {
            const uint32_t b = (f & 1) * 2 + ((f >> 1) & 1), k_addr = smem_u32(smem + L::kK + (f & 1) * kDbTile);
            mbar_wait_quiet(&k_full[f & 1], (f >> 1) & 1);
            mbar_wait_quiet(&s_free[b], ((f >> 2) & 1) ^ 1);
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < 4; ++i) umma_f16_ts(tmem_base + b * 64, t_q + i * 8, make_smem_desc_sw128(k_addr + i * 32), idesc, i != 0 ? 1u : 0u);
            umma_commit(&s_full[b]);
            umma_commit(&k_empty[f & 1]);
          }
          umma_commit(&q_free[k & 1]);
        }
      }
      __syncwarp();
    } else if (warp == 2) {
      // ============================== P V ==============================
      if (elect_one()) {
        constexpr uint32_t idesc = make_idesc_bmn(128, 64);
        uint32_t f = 0, n_v = 0;
        for (uint32_t k = 0;; ++k) {
          const DbItem it = db_item(smem, tab_full, k);
          mbar_arrive(&tab_empty[k & 1]);
          if (it.head < 0) break;
          for (int t = 0; t < it.tiles; ++t, ++f) {
            const uint32_t b = (f & 1) * 2 + ((f >> 1) & 1);
            mbar_wait_quiet(&p_ready[b], (f >> 2) & 1);
            mbar_arrive(&s_free[b]);
          }
          for (int j = 0; j < it.blocks(); ++j, ++f, ++n_v) {
            const uint32_t b = (f & 1) * 2 + ((f >> 1) & 1), s = n_v % kDbStages, v_addr = smem_u32(smem + L::kV + s * kDbTile);
            const uint32_t t_o = tmem_base + kDbTmemO + (f & 1) * 64, t_p = tmem_base + b * 64;
            // keys behind the end of the sequence belong to another one: groups of 16 of them stay out, as in the causal forward
            const int steps = min(4, (it.len - j * kDbBN + 15) / 16);
            mbar_wait_quiet(&v_full[s], (n_v / kDbStages) & 1);
            mbar_wait_quiet(&p_ready[b], (f >> 2) & 1);
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (i < steps) umma_f16_ts(t_o, t_p + i * 8, make_smem_desc_sw128_mn(v_addr + i * 16 * 128, kDbTile), idesc, j < 2 && i == 0 ? 0u : 1u);
            umma_commit(&s_free[b]);
            umma_commit(&pv_done[f & 1]);
            umma_commit(&v_empty[s]);
          }
        }
      }
      __syncwarp();
    } else {
      // ============================== items ==============================
      // sequences in the order of their number of blocks, the longest first; heads vary fastest
      const int* cu = p.cu_seqlens;
      auto blocks_of = [&](int s) { return (cu[s + 1] - cu[s] + kDbBM - 1) / kDbBM; };
      int level = 0, above = 0, upto = 0;      // row blocks of sequences that have more than `level` blocks, that many or more
      for (int s = lane; s < p.num_seqs; s += 32) level = max(level, blocks_of(s));
      level = __reduce_max_sync(0xffffffffu, level) + 1;
      for (uint32_t k = 0;; ++k) {
        const int at = (k & 1) ? (k + 1) * gridDim.x - 1 - blockIdx.x : k * gridDim.x + blockIdx.x;
        const int rank = at / p.heads;
        while (level > 0 && rank >= upto) {
          --level;
          above = upto;
          int n = 0;
          for (int s = lane; s < p.num_seqs; s += 32) n += blocks_of(s) == level ? level : 0;
          upto += __reduce_add_sync(0xffffffffu, n);
        }
        int e[6] = {-1, 0, 0, 0, 0, 0};
        if (level > 0 && rank < upto) {
          int n = (rank - above) / level;        // the n-th sequence of this many blocks
          e[1] = (rank - above - n * level) * kDbBM;
          for (int s0 = 0; s0 < p.num_seqs; s0 += 32) {
            const int s = s0 + lane;
            const bool has = s < p.num_seqs && blocks_of(s) == level;
            const uint32_t m = __ballot_sync(0xffffffffu, has);
            const uint32_t hit = __ballot_sync(0xffffffffu, has && __popc(m & ((1u << lane) - 1)) == n);
            if (hit != 0) {
              const int src = s0 + __ffs(hit) - 1;
              e[0] = at - rank * p.heads;
              e[2] = cu[src];
              e[3] = cu[src + 1] - cu[src];
              break;
            }
            n -= __popc(m);
          }
          e[4] = p.bucket(e[1] - (e[3] - 1)) >> 6;
          e[5] = max((p.bucket(min(e[1] + kDbBM, e[3]) - 1) >> 6) - e[4], 0) + 1;
        }
        db_wait_idle<1000>(&tab_empty[k & 1], ((k >> 1) & 1) ^ 1);
        if (lane == 0) {
          int* t = reinterpret_cast<int*>(smem + L::kTab + (k & 1) * 32);
#pragma unroll
          for (int i = 0; i < 6; ++i) t[i] = e[i];
          mbar_arrive(&tab_full[k & 1]);
        }
        __syncwarp();
        if (e[0] < 0) break;
      }
    }
  } else if (warp < 20) {
    // ============================== softmax, epilogue ==============================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
    const uint32_t w = (warp - 4) >> 3;                        // tiles w, w + 2, ...
    const int h = ((warp - 4) >> 2) & 1;                       // columns 32 h .. 32 h + 31 of a tile
    const int quad = warp & 3, r = quad * 32 + lane;           // row of the item == TMEM lane
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t a_row = smem_u32(smem + L::kA) + r * kDbAPitch;
    const uint32_t pair = 2 + w * 4 + quad;                    // barrier of the two warps that hold the same rows of a tile
    const int y0 = 127 - r;
    const uint32_t lut_off = L::kLut + (y0 & 1) * L::kLutCopy + (y0 & ~1) * 2 + h * 64;
    uint32_t f = 0, n_b = 0, n_pv = 0;                         // tiles of all items, key blocks of all items, P V of this stream
    for (uint32_t k = 0;; ++k) {
      const DbItem it = db_item(smem, tab_full, k);
      __syncwarp();
      if (lane == 0) mbar_arrive(&tab_empty[k & 1]);
      if (it.head < 0) break;
      // ---- A ----
      for (int t = 0; t < it.tiles; ++t, ++f) {
        if ((f & 1) != w) continue;
        const uint32_t b = w * 2 + ((f >> 1) & 1);
        mbar_wait_quiet(&s_full[b], (f >> 2) & 1);
        tc_fence_after();
        uint32_t sv[32];
        tmem_ld_32x32b_x32(t_lane + b * 64 + h * 32, sv);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[b]);
        const uint32_t dst = a_row + (it.tile0 + t) * 128 + h * 64;
#pragma unroll
        for (int i = 0; i < 16; ++i) sts_u32(dst + i * 4, pack_bf16x2(__uint_as_float(sv[i * 2]), __uint_as_float(sv[i * 2 + 1])));
      }
      named_barrier_sync(1, 512);
      // ---- keys ----
      float m_run = -INFINITY, l_run = 0.f;
      bool first = true;
      const int n = it.blocks();
      for (int j = 0; j < n; ++j, ++f, ++n_b) {
        if ((f & 1) != w) continue;
        const uint32_t b = w * 2 + ((f >> 1) & 1), s = n_b % kDbStages, t_s = t_lane + b * 64;
        const uint8_t* stage = smem + L::kB + s * L::kStage;
        const uint32_t st = smem_u32(stage);
        db_wait_block(st + L::kMeta + 36, n_b);
        mbar_wait_quiet(&b_full[s], (n_b / kDbStages) & 1);
        const uint4 g4 = *reinterpret_cast<const uint4*>(stage + L::kMeta + h * 16);
        const int flat = *reinterpret_cast<const int*>(stage + L::kMeta + 32);
        mbar_wait_quiet(&s_full[b], (f >> 2) & 1);
        tc_fence_after();
        uint32_t sv[32];
        tmem_ld_32x32b_x32(t_s + h * 32, sv);
        tmem_ld_wait();
        // the streams take turns at the lookups, which are bound by shared memory, so that one looks up while the other forms its weights
        if (j > 0) named_barrier_sync(10 + w, 512);
        float a0 = 0.f;
        if (flat >= 0) {
          a0 = add_lds_bf16(0.f, a_row + flat * 2);
          db_add_column(sv, st + (flat & 7) * 2 + h * (32 * 16));
        } else {
          const uint32_t b_row[4] = {g4.x, g4.y, g4.z, g4.w};
          db_add_tables(sv, st + lut_off, a_row, b_row);
        }
        if (j + 1 < n) asm volatile("bar.arrive %0, 512;" ::"r"(10 + (w ^ 1)) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_empty[s]);
        const int see = it.len - j * kDbBN - h * 32;           // keys of this half
        if (see < 32) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i >= see) sv[i] = 0xff800000u;
        }
        // ---- online softmax ----
        float mx2[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 32; i += 2) mx2[(i >> 1) & 1] = fmaxf(mx2[(i >> 1) & 1], fmaxf(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])));
        const float mx = (fmaxf(mx2[0], mx2[1]) + a0) * p.scale_log2;
        // The row's own maximum: the larger of both halves, which also orders their reads of the scores before the first P over them.  A stale one would do for the
        // range (a weight below 2^8 is harmless), but a row's largest weight has to be exactly 1 to pass the rounding of P whole
        const uint32_t t_mx = t_lane + kDbTmemMax + w * 4 + (n_pv & 1) * 2;
        tmem_st_x1(t_mx + h, __float_as_uint(mx));
        tmem_st_wait();
        tc_fence_before();
        named_barrier_sync(pair, 64);
        tc_fence_after();
        const float both = tmem_max_x2(t_mx);
        const bool moved = both > m_run;
        float corr = 1.f;
        if (moved) {
          corr = ex2_approx(m_run - both);
          m_run = both;
        }
        if (__any_sync(0xffffffffu, moved && !first)) {
          mbar_wait_quiet(&pv_done[w], (n_pv - 1) & 1);
          tc_fence_after();
          uint32_t ov[32];
          tmem_ld_32x32b_x32(t_lane + kDbTmemO + w * 64 + h * 32, ov);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
          tmem_st_32x32b_x32(t_lane + kDbTmemO + w * 64 + h * 32, ov);
        }
        const float m_sub = m_run == -INFINITY ? 0.f : m_run, off = fmaf(a0, p.scale_log2, -m_sub);
        const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2), off2 = pack_f32x2(off, off);
        uint64_t sum2[2] = {0, 0};
        uint32_t pv[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float a, c;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sc2, off2), a, c);
          a = ex2_approx(a);
          c = ex2_approx(c);
          pv[i / 2] = pack_bf16x2(a, c);
          sum2[(i >> 1) & 1] = add_f32x2(sum2[(i >> 1) & 1], pack_f32x2(a, c));
        }
        tmem_st_32x32b_x16(t_s + h * 16, pv);
        float s0, s1;
        unpack_f32x2(add_f32x2(sum2[0], sum2[1]), s0, s1);
        l_run = l_run * corr + (s0 + s1);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[b]);
        first = false;
        ++n_pv;
      }
      // ---- both streams' O, 16 columns per warpgroup; one of them is empty where there is one block of keys ----
      if (!first) mbar_wait_quiet(&pv_done[w], (n_pv - 1) & 1);
      tmem_st_x2(t_lane + kDbTmemML + (w * 2 + h) * 2, __float_as_uint(m_run), __float_as_uint(l_run));
      tmem_st_wait();
      tc_fence_before();
      named_barrier_sync(1, 512);
      tc_fence_after();
      const uint32_t col = w * 32 + h * 16;
      uint32_t ml[8], o0[16], o1[16];
      tmem_ld_32x32b_x8(t_lane + kDbTmemML, ml);
      tmem_ld_32x32b_x16(t_lane + kDbTmemO + col, o0);
      tmem_ld_32x32b_x16(t_lane + kDbTmemO + 64 + col, o1);
      tmem_ld_wait();
      tc_fence_before();                                       // the next item's P V follows the barrier behind its A
      const float m0 = __uint_as_float(ml[0]), m1 = __uint_as_float(ml[4]), m_all = fmaxf(m0, m1);
      float f0 = ex2_approx(m0 - m_all), f1 = ex2_approx(m1 - m_all);
      const float inv = 1.f / ((__uint_as_float(ml[1]) + __uint_as_float(ml[3])) * f0 + (__uint_as_float(ml[5]) + __uint_as_float(ml[7])) * f1);
      f0 *= inv;
      f1 *= inv;
      const int row = it.q0 + r;
      if (row < it.len) {
        const bool empty0 = n == 1 && first == (w == 0), empty1 = n == 1 && first == (w == 1);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (empty0) o0[i] = 0u;
          if (empty1) o1[i] = 0u;
        }
        __nv_bfloat16* orow = p.out + (it.start + row) * p.o_stride_t + it.head * 64 + col;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          o0[i] = pack_bf16x2(fmaf(__uint_as_float(o0[2 * i]), f0, __uint_as_float(o1[2 * i]) * f1),
                              fmaf(__uint_as_float(o0[2 * i + 1]), f0, __uint_as_float(o1[2 * i + 1]) * f1));
        stg_v8(orow, o0);
      }
      __syncwarp();
    }
  } else {
    // ============================== queries, buckets, B ==============================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    const int quad = warp & 3, r = quad * 32 + lane;
    auto queries = [&](uint32_t k) {
      const DbItem it = db_item(smem, tab_full, k);
      __syncwarp();
      if (it.head < 0) return it;
      uint32_t qv[32];
      const int row = it.q0 + r;
      const uint4* src = reinterpret_cast<const uint4*>(p.q + (it.start + row) * p.q_stride_t + it.head * 64);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint4 v = row < it.len ? __ldg(src + i) : make_uint4(0, 0, 0, 0);
        qv[4 * i] = v.x; qv[4 * i + 1] = v.y; qv[4 * i + 2] = v.z; qv[4 * i + 3] = v.w;
      }
      db_wait_idle<100>(&q_free[k & 1], ((k >> 1) & 1) ^ 1);
      tc_fence_after();
      tmem_st_32x32b_x32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + kDbTmemQ + (k & 1) * 32, qv);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_ready[k & 1]);
      return it;
    };
    uint32_t n_b = 0;
    DbItem next = queries(0);
    for (uint32_t k = 0;; ++k) {
      const DbItem it = next;
      if (lane == 0) mbar_arrive(&tab_empty[k & 1]);
      if (it.head < 0) break;
      next = queries(k + 1);
      const int row0 = it.head * p.total_tokens + it.start;                   // of this sequence in the table
      for (int j = 0; j < it.blocks(); ++j, ++n_b) {
        const uint32_t s = n_b % kDbStages;
        if (s != static_cast<uint32_t>(quad)) continue;
        const int key0 = j * kDbBN, first = it.q0 - key0 + kDbBM - 1;         // entry y is the bucket of first - y; row r and key c: y = 127 - r + c
        int c[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) c[i] = p.bucket(first - (i * 32 + lane));
        const int c_lo = p.bucket(it.q0 - key0 - (lane & 7) * 8 - 7) & ~7;    // lane g < 8: lowest column of its 8 keys
        const int c_max = __shfl_sync(0xffffffffu, c[0], 0), c_min = __shfl_sync(0xffffffffu, c[5], 30);
        const bool flat = c_max == c_min;
        db_wait_idle<40>(&b_empty[s], ((n_b / kDbStages) & 1) ^ 1);
        uint8_t* st = smem + L::kB + s * L::kStage;
        if (lane == 0) mbar_arrive_expect_tx(&b_full[s], flat ? kDbBN * 16 : kDbBN * kDbWin * 2);
        __syncwarp();
        if (flat) {
          if (lane == 0) tma_load_2d(st, &tmB1, &b_full[s], c_min & ~7, row0 + key0);
        } else if (lane < 8) {
          tma_load_2d(st + lane * 8 * kDbWin * 2, &tmB, &b_full[s], c_lo, row0 + key0 + lane * 8);
        }
        if (!flat) {
          const uint32_t lut = smem_u32(st + L::kLut);
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            const int y = i * 32 + lane;
            sts_u16(lut + y * 2, c[i] * 2);
            if (y > 0) sts_u16(lut + L::kLutCopy + (y - 1) * 2, c[i] * 2);
          }
        }
        int* meta = reinterpret_cast<int*>(st + L::kMeta);
        if (lane < 8) meta[lane] = static_cast<int>(smem_u32(st)) + (lane >> 2) * (32 * kDbWin * 2) - 2 * c_lo;
        if (lane == 8) meta[8] = flat ? c_min : -1;
        if (lane == 9) meta[9] = n_b;
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_full[s]);
      }
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

// maps = {position keys [NB, H * 64], K, V (boxes 64 x 64, sw128), B [H * T, NB] box 8 x 144, the same box 64 x 8 (no swizzle)}
extern "C" cudaError_t nrl_deberta_attn_tc(const CUtensorMap* maps, const void* q, long q_stride_t, void* out, long o_stride_t, const int* cu, int num_seqs,
                                           int total, int heads, float scale, const short* lut, int lut_center, int buckets, int num_sms, cudaStream_t s) {
  using namespace nrl;
  if (total == 0 || num_seqs == 0) return cudaSuccess;
  if (buckets > kDbMaxBuckets || buckets < 1) return cudaErrorInvalidValue;
  DbParams p;
  p.cu_seqlens = cu; p.q = static_cast<const __nv_bfloat16*>(q); p.out = static_cast<__nv_bfloat16*>(out); p.lut = lut;
  p.q_stride_t = q_stride_t; p.o_stride_t = o_stride_t; p.num_seqs = num_seqs; p.total_tokens = total; p.heads = heads;
  p.lut_center = lut_center; p.buckets = buckets; p.scale_log2 = scale * 1.4426950408889634f;
  const cudaError_t e = cudaFuncSetAttribute(deberta_attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DbSmem::kTotal);
  if (e != cudaSuccess) return e;
  const long most = static_cast<long>(total / kDbBM + num_seqs) * heads;
  launch_dependent(deberta_attn_tc_kernel, static_cast<int>(most < num_sms ? most : num_sms), kDbThreads, DbSmem::kTotal, s, maps[0], maps[1], maps[2], maps[3],
                   maps[4], p);
  return cudaGetLastError();
}
