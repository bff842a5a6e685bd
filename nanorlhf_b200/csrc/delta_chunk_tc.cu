// Gated delta rule (or plain accumulation) of prompt portions with one decay per head, 32 tokens at a time on tcgen05 / TMEM.
// With g_i the decays of a chunk, c_i = g_1 .. g_i and G(i, j) = g_{j+1} .. g_i (products, nothing is divided), over the state S before it:
//   u_i = beta_i (v_i - c_i S^T k_i - sum_{j<i} G(i,j) (k_i . k_j) u_j)          (no delta: u_i = v_i)
//   o_i = c_i S^T q_i + sum_{j<=i} G(i,j) (q_i . k_j) u_j
//   S  <- c_n S + sum_j G(n,j) k_j u_j^T
// The four products (S^T [K; Q], [K; Q] K^T, S^T += U K, U (Q K^T)) run on the tensor cores and nothing is held in less than float: every float operand is the
// sum of three bf16 terms (8 + 8 + 8 bits and their signs, so exact to its last bit), a product is the six pairs of terms above 2^-24, and
// all pairs but first x first are summed first.  The tensor cores cut their sums off where float arithmetic rounds (64 products in one accumulator: 6.5e-8
// relative to float64, float32 sums 5.1e-8), so at most 64 products of first terms go into one accumulator; the state itself stays in float registers
// (one rounding per chunk), products of decays carry two floats, and what earlier tokens take off u is summed by itself.  Error against float64, 16 x 2048
// tokens, 16 heads of 128 x 128: outputs 1.29e-7, state 7.8e-8; four tokens at a time in float 1.34e-7, 1.04e-7.
//
// Block per (entry, head, 128 columns of the state): TMEM lanes are columns of S, so the triangular solve is each thread's own.
//   warps 0..3    solve: thread per column; u into TMEM as the next products' A operand, outputs
//   warps 4..11   state: two threads per column, 64 rows each in registers; sum of the chunk, new terms into TMEM
//   warps 12..15  terms of q and k into 128B-swizzled tiles
//   warps 16..19  the two masked 32 x 32 Gram matrices
//   warp 20       issues the MMAs
//   warp 21       brings q, k and v two chunks ahead, a row per bulk copy (21..23 float by float where rows are not aligned)
// Chain per chunk: terms of S -> S^T K -> solve -> U K -> S; S^T Q and the Gram products of the next chunk run beside the solve.
//
// 16 x 2048 tokens, 16 heads of 128 x 128 (two rounds of blocks): 630 us, 2290 four tokens at a time; one portion of 1000: 158 / 733.  A chunk takes 8700
// clocks: solve 2500 (its 496 multiply-adds a thread read the Gram matrix by broadcasts, 254 KB of shared-memory returns at 128 bytes a clock), sum and terms of
// S 2800, S^T K and its read-out 2200, U K 1100; the MMAs alone would take 4200, and the schedulers issue in 64 % of the clocks.  The code is kept small,
// in loops where nothing waits for them, since every warp runs through its part once per chunk: at 100 KB of code the SMs wait for
// instructions together (16 blocks 160 us, 256 blocks 1000 us of the same work each; at 75 KB both take the same time per chunk).
// Compiled WITHOUT fast-math.
#include "attention_tc.cuh"
#include "hybrid_kernels.h"

#include <algorithm>
#include <functional>
#include <vector>

namespace nrl {
namespace {

constexpr int kC = 32;                          // tokens of a chunk
constexpr int kDcThreads = 24 * 32;         // registers: 768 x 80 at launch = 128 x (104 + 112 + 112 + 56 + 56 + 40)
constexpr int kDcLoaders = 96;                  // threads that copy single floats
constexpr int kDcTile = 2 * kC * 128;           // [K; Q]: 64 rows of 64 bf16, 128B-swizzled (8 KB)

template <int DP>
struct DcSmem {
  static constexpr int kHalves = DP / 64;
  static constexpr int kKQ = 0;                                         // [stage][term][half of the rows of S] tiles
  static constexpr int kKQStage = 3 * kHalves * kDcTile;
  static constexpr int kM = kKQ + 2 * kKQStage;                         // [stage] Q K^T: terms 0 | 1 side by side in one tile, 2 in another
  static constexpr int kMStage = 2 * kC * 128;
  static constexpr int kL = kM + 2 * kMStage;                           // [stage][j][i] floats: beta_i G(i,j) k_i . k_j
  static constexpr int kLStage = kC * kC * 4;
  static constexpr int kSc = kL + 2 * kLStage;                          // [stage] beta | c | G(n, .) | g | ones
  static constexpr int kScStage = 5 * kC * 4;
  static constexpr int kRaw = kSc + 2 * kScStage;                       // [stage] K | Q [32][DP] floats, V [32][128] floats
  static constexpr int kRawV = 2 * kC * DP * 4;
  static constexpr int kRawStage = kRawV + kC * 128 * 4;
  static constexpr int kBar = kRaw + 2 * kRawStage;
  static constexpr int kUsed = kBar + 256;
  static constexpr int kTotal = kUsed > 116 * 1024 ? kUsed : 116 * 1024;      // TMEM: one block per SM
};

// TMEM columns.  The terms of S, and once S^T [K; Q] is formed the scaled terms of U and the sum for S in their place: per half of
// the rows 96 columns of terms, or 64 of the sum and a part of U's terms behind them.
template <int DP>
struct DcTmem {
  static constexpr int kHalf = 96;
  __device__ static constexpr int uh(int term) { return DP == 128 ? (term < 2 ? 64 + 16 * term : 160) : 64 + 16 * term; }
  static constexpr int kR1 = 192, kR2 = 256;                // S^T [K; Q] in two accumulators: first terms of the upper rows in the second
  static constexpr int kO2 = 320;
  static constexpr int kU = 352;                            // + 16 term
  static constexpr int kG1 = 416, kG2 = 448;                // Gram, likewise
};

NRL_DEVICE void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// product of two numbers that are each the sum of two floats
NRL_DEVICE float2 mul_wide(float2 a, float2 b) {
  const float p = a.x * b.x;
  return make_float2(p, fmaf(a.x, b.x, -p) + fmaf(a.x, b.y, a.y * b.x));
}

// as umma_f16, umma_f16_ts and umma_commit, by the lane that has `leader` set
NRL_DEVICE void dc_mma(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate),
      "r"(leader)
      : "memory");
}
NRL_DEVICE void dc_mma_ts(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate),
      "r"(leader)
      : "memory");
}
NRL_DEVICE void dc_commit(uint32_t leader, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(smem_u32(bar)), "r"(leader)
      : "memory");
}

// two floats as three pairs of bf16 whose sum they are
NRL_DEVICE void split3(float a, float b, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
  const uint64_t minus1 = pack_f32x2(-1.f, -1.f);
  t0 = pack_bf16x2(a, b);
  unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(t0 << 16), __uint_as_float(t0 & 0xffff0000u)), minus1, pack_f32x2(a, b)), a, b);
  t1 = pack_bf16x2(a, b);
  unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(t1 << 16), __uint_as_float(t1 & 0xffff0000u)), minus1, pack_f32x2(a, b)), a, b);
  t2 = pack_bf16x2(a, b);
}

// one float, zero unless `ok`
NRL_DEVICE void cp_async_zfill(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
NRL_DEVICE void bulk_load(float* dst, const float* src, uint32_t bytes, uint64_t* bar) {      // 16-byte aligned, a multiple of 16 bytes
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes),
               "r"(smem_u32(bar))
               : "memory");
}

// pairs of terms of a product, the small ones first: (0,2) (1,1) (2,0) (0,1) (1,0) (0,0)
NRL_DEVICE int pair_a(int pr) { return (0x010210 >> (4 * pr)) & 3; }
NRL_DEVICE int pair_b(int pr) { return (0x001012 >> (4 * pr)) & 3; }

// More items (entry, head, 128 columns) than SMs: their chunks lie on a line, entry by entry, and block j takes the `per` chunks of it from j per on, an even share or
// the longest item.  An item that a block's end cuts is computed first by the block behind, at that block's start (its first chunks, as many as lie there
// on the line), and then by this block, at its end, from the state that the other has left: no item is longer than `per`, so that state is there by then.
// Blocks take their places from the line's end in the order in which they start (a ticket), so that none waits for one that has not started; should the wait run out
// all the same, the state becomes NaN.
// The segments are laid out by a kernel of their own, and between two segments the block starts anew (barriers and all): code that every warp runs through is
// dear here.  With phases that run on over the segments a chunk took 19 % longer, so 13 % (92 KB of code, 78 for whole items).
// 10 x 2048 tokens, 16 heads of 128 x 128 (160 items of 64 chunks on 148 SMs): two rounds of 64 chunks 625 us, 70 chunks in a row 381 us.
// Whether it pays depends on the lengths: no block gets less than the longest item, and whole items of unequal lengths do not run in rounds.  The line is taken where
// it is estimated a tenth below the least that whole items can take: an SM has r items of length l and more wherever more than (r - 1) SMs' worth of them exist.  A
// caller who has the lengths on the host asks there (nrl_delta_line_pays); for others the kernel that lays the segments out decides.  16 heads, one entry of 4000
// tokens and nine of 400: whole 600 us, line 768; 8 heads of 64, 20 entries of 33 to 700: 100 / 181.
struct DcSegment {
  int t0, n, t1;              // first token, chunks, end of the entry's tokens
  int h, cb0, e;              // head, first column, entry
  int in, out;                // the state comes from the block behind / goes to the block in front
};
struct DcLine {
  DcSegment* segments;        // [items + blocks]
  int *first, *last;          // [blocks] a block's segments
  int* handed;                // [blocks] 1 once the state that the block hands on is there
  float* carry;               // [blocks][128][128]
  int* taken;                 // [1] the line is taken, else a block has an item
  int* ticket;                // [1] blocks that have started
};
constexpr int kDcMaxEntries = 4096;

// chunks in a row of the line against those of whole items; a chunk costs 13 % more there, starting anew between segments about four chunks
__host__ NRL_DEVICE bool line_pays(long line, long whole) { return 113 * line + 400 < 90 * whole; }

__global__ void __launch_bounds__(1024) delta_line_kernel(const int* __restrict__ cu, int E, int heads, int parts, int blocks, bool forced, const DcLine l) {
  __shared__ int from[kDcMaxEntries + 1];                  // chunks of an item of the entries in front
  __shared__ int most[32], least[32];
  const int tid = threadIdx.x, items = heads * parts;
  for (int b = tid; b < blocks; b += blockDim.x) l.first[b] = l.last[b] = l.handed[b] = 0;
  auto chunks = [&](int e) { return max(1, (cu[e + 1] - cu[e] + kC - 1) / kC); };      // an entry without tokens keeps its state: one empty chunk
  int m = 0;
  for (int e = tid; e < E; e += blockDim.x) m = max(m, chunks(e));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((tid & 31) == 0) most[tid >> 5] = m;
  if (tid < 32) {
    int base = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      int upto = e0 + tid < E ? chunks(e0 + tid) : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, upto, d);
        if (tid >= d) upto += y;
      }
      if (e0 + tid < E) from[e0 + tid + 1] = base + upto;
      base += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (tid == 0) from[0] = 0;
  }
  __syncthreads();
  m = most[tid & 31];
  const int total = from[E] * items, share = (total + blocks - 1) / blocks, per = max(__reduce_max_sync(0xffffffffu, m), share);
  int whole = share;
  for (int e = tid; e < E && !forced; e += blockDim.x) {   // at most a few hundred entries where the line comes into question
    const int n = from[e + 1] - from[e];
    int as_long = 0;
    for (int k = 0; k < E; ++k) as_long += from[k + 1] - from[k] >= n ? 1 : 0;
    whole = max(whole, (as_long * items + blocks - 1) / blocks * n);
  }
  whole = __reduce_max_sync(0xffffffffu, whole);
  if ((tid & 31) == 0) least[tid >> 5] = whole;
  __syncthreads();
  whole = __reduce_max_sync(0xffffffffu, least[tid & 31]);
  const bool taken = forced || line_pays(per, whole);
  if (tid == 0) {
    *l.taken = taken ? 1 : 0;
    *l.ticket = 0;
  }
  if (!taken) return;
  for (int q = tid; q < E * items; q += blockDim.x) {
    const int e = q / items, k = q - e * items, n = from[e + 1] - from[e], s = from[e] * items + k * n, t0 = cu[e], t1 = cu[e + 1];
    const int h = k / parts, cb0 = (k - h * parts) * 128, a = s / per, here = min(n, (a + 1) * per - s);      // chunks that lie in block a
    l.segments[q + a] = DcSegment{t0 + (n - here) * kC, here, t1, h, cb0, e, here < n, 0};
    if (s == a * per) l.first[a] = q + a;
    if (s + n >= (a + 1) * per || q == E * items - 1) l.last[a] = q + a + 1;
    if (here < n) {                                        // the rest, which is computed first
      l.segments[q + a + 1] = DcSegment{t0, n - here, t1, h, cb0, e, 0, 1};
      l.first[a + 1] = q + a + 1;
      if (s + n >= (a + 2) * per || q == E * items - 1) l.last[a + 1] = q + a + 2;
    }
  }
}

// has the state been handed on (by a whole warp); false after some seconds
NRL_DEVICE bool dc_handed(const int* flag) {
  int ok = 0;
  for (int n = 0; ok == 0 && n < (1 << 22); ++n) {
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(ok) : "l"(flag) : "memory");
    if (ok == 0) __nanosleep(500);
  }
  return __all_sync(0xffffffffu, ok != 0);
}

struct DcParams {
  const float *qkv, *beta, *decay;
  float *state, *o;
  const int *cu, *start, *state_slot;
  long sq;
  int col_k, col_v, heads, kv_heads, D, Dv;
  DcLine line;
};

NRL_DEVICE void mbar_inval(uint64_t* bar) { asm volatile("mbarrier.inval.shared.b64 [%0];" ::"r"(smem_u32(bar)) : "memory"); }

// DP: padded rows of S; WIDE: rows of q, k and v are 16-byte aligned; LINE: a block takes its share of the line instead of an item.  Where the GPU decides, both
// kernels are launched and one of them finds nothing to do: 10 entries of 2048 tokens 396 us (388 with the lengths on the host), 20 of 33 to 700 110 us (100).  Both
// forms in one kernel spill: 401 and 105.
template <int DP, bool DELTA, bool WIDE, bool LINE>
__global__ void __launch_bounds__(kDcThreads, 1) delta_chunk_tc_kernel(const DcParams p) {
  if (!LINE && p.line.taken != nullptr && *p.line.taken != 0) return;
  using L = DcSmem<DP>;
  using Tm = DcTmem<DP>;
  constexpr int NH = L::kHalves;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* kq_full = reinterpret_cast<uint64_t*>(smem + L::kBar);      // [stage] tiles, beta and decays of a chunk are here
  uint64_t* kq_free = kq_full + 2;                                      // [stage] the MMAs have read them
  uint64_t* lm_full = kq_free + 2;                                      // [stage] Gram matrices
  uint64_t* sc_free = lm_full + 2;                                      // [stage] solve, state and Gram warps are done with the Gram matrix and the scalars
  uint64_t* gram_full = sc_free + 2;
  uint64_t* gram_free = gram_full + 1;
  uint64_t* raw_full = gram_free + 1;                                   // [stage]
  uint64_t* raw_free = raw_full + 2;                                    // [stage]
  uint64_t* sp_full = raw_free + 2;                                     // [16 rows of each half] terms of S
  uint64_t* rk_full = sp_full + 4;                                      // S^T K
  uint64_t* rq_full = rk_full + 1;                                      // S^T Q
  uint64_t* uh_full = rq_full + 1;                                      // scaled terms of U
  uint64_t* u_full = uh_full + 1;                                       // terms of U; S^T [K; Q] has been read
  uint64_t* ds_full = u_full + 1;                                       // sum for S
  uint64_t* o2_full = ds_full + 1;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(o2_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto init_barriers = [&]() {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kq_full[i], 128);
      mbar_init(&kq_free[i], 1);
      mbar_init(&lm_full[i], 128);
      mbar_init(&sc_free[i], 512);
      mbar_init(&raw_full[i], WIDE ? 32 : kDcLoaders);
      mbar_init(&raw_free[i], 256);
    }
    for (int i = 0; i < 4; ++i) mbar_init(&sp_full[i], 256);
    mbar_init(gram_full, 1);
    mbar_init(gram_free, 128);
    mbar_init(rk_full, 1);
    mbar_init(rq_full, 1);
    mbar_init(uh_full, 128);
    mbar_init(u_full, 128);
    mbar_init(ds_full, 1);
    mbar_init(o2_full, 1);
    fence_mbar_init();
  };
  volatile int* ticket = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  if (warp == 20) {
    if (lane == 0) {
      init_barriers();
      if (LINE) *ticket = atomicAdd(p.line.ticket, 1);
    }
    __syncwarp();
    tmem_alloc(tmem_ptr, 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;

  const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
  auto line = [&]() { return static_cast<int>(gridDim.x) - 1 - *ticket; };      // this block's place, read again rather than kept
  const int first = LINE ? p.line.first[line()] : 0, last = LINE ? p.line.last[line()] : 1;      // segments of this block
  int e, h, cb0, t0, n_chunks, t1;
  auto take = [&](int i) {
    if (LINE) {
      const DcSegment& sg = p.line.segments[i];
      e = sg.e; h = sg.h; cb0 = sg.cb0; t0 = sg.t0; n_chunks = sg.n; t1 = sg.t1;
    } else {
      const unsigned parts = (p.Dv + 127) / 128, eh = blockIdx.x / parts;
      e = static_cast<int>(eh / p.heads);
      h = static_cast<int>(eh % p.heads);
      cb0 = static_cast<int>(blockIdx.x % parts) * 128;
      t0 = p.cu[e];
      t1 = p.cu[e + 1];
      n_chunks = (t1 - t0 + kC - 1) / kC;
    }
  };
  if (!LINE) take(0);
  // between two segments: everybody has done with the barriers, then they start anew
  auto turn = [&]() {
    if (!LINE) return;
    __syncwarp();
    tc_fence_before();
    named_barrier_sync(3, kDcThreads);
    if (warp == 20 && lane == 0) {
      for (uint64_t* b = kq_full; b <= o2_full; ++b) mbar_inval(b);
      init_barriers();
    }
    named_barrier_sync(3, kDcThreads);
    tc_fence_after();
  };

  if (warp < 4) {
    // ============================== solve and outputs ==============================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
#pragma unroll 1
    for (int i = first; i < last; ++i, turn()) {
      if (LINE) take(i);
      for (int n = 0; n < n_chunks; ++n) {
        const int st = n & 1;
        const uint32_t ph = n & 1, ph2 = (n >> 1) & 1;
        const float* sc = reinterpret_cast<const float*>(smem + L::kSc + st * L::kScStage);
        float u[kC], r[kC];
        mbar_wait_quiet(&raw_full[st], ph2);
        const float* v = reinterpret_cast<const float*>(smem + L::kRaw + st * L::kRawStage + L::kRawV) + (warp & 3) * 32 + lane;
#pragma unroll
        for (int i = 0; i < kC; ++i) u[i] = v[i * 128];
        mbar_arrive(&raw_free[st]);
        mbar_wait_quiet(&kq_full[st], ph2);
        mbar_wait_quiet(rk_full, ph);
        tc_fence_after();
        auto read_rq = [&](int c, uint32_t (&a)[16]) {       // sixteen columns of S^T [K; Q]
          tmem_ld_32x32b_x16(tmem + Tm::kR1 + c + lane_off, a);
          uint32_t b[16];
          tmem_ld_32x32b_x16(tmem + Tm::kR2 + c + lane_off, b);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
        };
        if (DELTA) {
#pragma unroll
          for (int c = 0; c < kC; c += 16) {
            uint32_t x[16];
            read_rq(c, x);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 b4 = *reinterpret_cast<const float4*>(sc + c + i), c4 = *reinterpret_cast<const float4*>(sc + kC + c + i);
              u[c + i] = b4.x * (u[c + i] - c4.x * __uint_as_float(x[i]));
              u[c + i + 1] = b4.y * (u[c + i + 1] - c4.y * __uint_as_float(x[i + 1]));
              u[c + i + 2] = b4.z * (u[c + i + 2] - c4.z * __uint_as_float(x[i + 2]));
              u[c + i + 3] = b4.w * (u[c + i + 3] - c4.w * __uint_as_float(x[i + 3]));
            }
          }
          mbar_wait_quiet(&lm_full[st], ph2);
          const float* lj = reinterpret_cast<const float*>(smem + L::kL + st * L::kLStage);
#pragma unroll
          for (int i = 0; i < kC; ++i) r[i] = 0.f;           // a sum of its own: smaller than u, and so are its roundings
#pragma unroll
          for (int j = 0; j < kC; ++j) {
            u[j] -= r[j];
#pragma unroll
            for (int i4 = (j + 1) / 4; i4 < kC / 4; ++i4) {
              const float4 w = *reinterpret_cast<const float4*>(lj + j * kC + i4 * 4);
              if (i4 * 4 + 0 > j) r[i4 * 4 + 0] = fmaf(w.x, u[j], r[i4 * 4 + 0]);
              if (i4 * 4 + 1 > j) r[i4 * 4 + 1] = fmaf(w.y, u[j], r[i4 * 4 + 1]);
              if (i4 * 4 + 2 > j) r[i4 * 4 + 2] = fmaf(w.z, u[j], r[i4 * 4 + 2]);
              if (i4 * 4 + 3 > j) r[i4 * 4 + 3] = fmaf(w.w, u[j], r[i4 * 4 + 3]);
            }
          }
        }
        mbar_wait_quiet(rq_full, ph);                                // the terms of S, which U's go over, have been read
        tc_fence_after();
        // Terms of U: scaled for the state, then as they are for the outputs.  The products of a row of U reach tokens before u_j with a weight of
        // zero: a value that is not finite would spoil them, so it is taken out in front of the second pass, and its token and all behind it
        // are made NaN at the output.
        int bad = kC;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
          if (pass == 1) {
            float probe = 0.f;
#pragma unroll
            for (int i = 0; i < kC; ++i) probe = fmaf(u[i], 0.f, probe);
            if (probe != probe) {
#pragma unroll
              for (int i = kC - 1; i >= 0; --i)
                if (!(fabsf(u[i]) < INFINITY)) {
                  bad = i;
                  u[i] = 0.f;
                }
            }
          }
          const float* ws = sc + (pass == 0 ? 2 : 4) * kC;   // G(n, .) or ones
          const uint32_t to = tmem + lane_off + (pass == 0 ? Tm::uh(0) : Tm::kU), third = pass == 0 ? Tm::uh(2) - Tm::uh(0) : 32;
#pragma unroll
          for (int c = 0; c < kC; c += 16) {
            uint32_t s0[8], s1[8], s2[8];
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 w = *reinterpret_cast<const float4*>(ws + c + i);
              split3(w.x * u[c + i], w.y * u[c + i + 1], s0[i / 2], s1[i / 2], s2[i / 2]);
              split3(w.z * u[c + i + 2], w.w * u[c + i + 3], s0[i / 2 + 1], s1[i / 2 + 1], s2[i / 2 + 1]);
            }
            tmem_st_32x32b_x8(to + c / 2, s0);
            tmem_st_32x32b_x8(to + 16 + c / 2, s1);
            tmem_st_32x32b_x8(to + third + c / 2, s2);
          }
          tmem_st_wait();
          tc_fence_before();
          if (pass == 0) mbar_arrive(uh_full);
        }
#pragma unroll
        for (int c = 0; c < kC; c += 16) {
          uint32_t x[16];
          read_rq(kC + c, x);
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 w = *reinterpret_cast<const float4*>(sc + kC + c + i);
            r[c + i] = w.x * __uint_as_float(x[i]);
            r[c + i + 1] = w.y * __uint_as_float(x[i + 1]);
            r[c + i + 2] = w.z * __uint_as_float(x[i + 2]);
            r[c + i + 3] = w.w * __uint_as_float(x[i + 3]);
          }
        }
        tc_fence_before();
        mbar_arrive(u_full);
        mbar_arrive(&sc_free[st]);
        if (LINE) take(i);                                     // looked up in every chunk, not kept
        const int t = t0 + n * kC, col = cb0 + (warp & 3) * 32 + lane;      // of S
        mbar_wait_quiet(o2_full, ph);
        tc_fence_after();
        float* od = p.o + (static_cast<long>(t) * p.heads + h) * p.Dv + col;
        const int left = col < p.Dv ? t1 - t : 0;
#pragma unroll
        for (int c = 0; c < kC; c += 16) {
          uint32_t x[16];
          tmem_ld_32x32b_x16(tmem + Tm::kO2 + c + lane_off, x);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (c + i < left) *od = c + i >= bad ? NAN : r[c + i] + __uint_as_float(x[i]);
            od += static_cast<long>(p.heads) * p.Dv;
          }
        }
        tc_fence_before();
      }
    }
  } else if (warp < 12) {
    // ============================== state ==============================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const int half = (warp - 4) >> 2;
#pragma unroll 1
    for (int i = first; i < last; ++i, turn()) {
      if (LINE) take(i);
      if (half < NH) {
        const int col = cb0 + (warp & 3) * 32 + lane;
        float* gS = p.state + ((static_cast<long>(p.state_slot[e]) * p.heads + h) * p.D + half * 64) * p.Dv + col;
        int rows = col < p.Dv ? p.D - half * 64 : 0;                                              // rows of S here
        int from = p.start[e] > 0 ? rows : 0;                                                     // rows that are carried
        float S[64];
        const float* ld = gS;
        long step = p.Dv;
        bool there = true;
        if (LINE && p.line.segments[i].in) {
          there = dc_handed(p.line.handed + line() + 1);
          ld = p.line.carry + (static_cast<long>(line() + 1) * 128 + half * 64) * 128 + (warp & 3) * 32 + lane;
          step = 128;
          from = rows;
        }
#pragma unroll
        for (int d = 0; d < 64; ++d, ld += step) S[d] = d < from ? __ldcg(ld) : 0.f;
        if (!there) S[0] = NAN;
        const uint32_t base = tmem + Tm::kHalf * half + lane_off;
        for (int n = 0; n < n_chunks; ++n) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t s0[8], s1[8], s2[8];
#pragma unroll
            for (int i = 0; i < 16; i += 2) split3(S[c * 16 + i], S[c * 16 + i + 1], s0[i / 2], s1[i / 2], s2[i / 2]);
            tmem_st_32x32b_x8(base + c * 8, s0);
            tmem_st_32x32b_x8(base + 32 + c * 8, s1);
            tmem_st_32x32b_x8(base + 64 + c * 8, s2);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&sp_full[c]);
          }
          mbar_wait_quiet(&kq_full[n & 1], (n >> 1) & 1);
          const float c_n = reinterpret_cast<const float*>(smem + L::kSc + (n & 1) * L::kScStage)[2 * kC - 1];
          mbar_arrive(&sc_free[n & 1]);
          mbar_wait_quiet(ds_full, n & 1);
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t x[16];
            tmem_ld_32x32b_x16(base + c * 16, x);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) S[c * 16 + i] = fmaf(c_n, S[c * 16 + i], __uint_as_float(x[i]));
          }
          tc_fence_before();
        }
        step = p.Dv;
        const bool out = LINE && p.line.segments[i].out;
        if (LINE) {                                          // the segment is looked up again: nothing of it is kept over the loop
          take(i);
          rows = cb0 + (warp & 3) * 32 + lane < p.Dv ? p.D - half * 64 : 0;
          gS = out ? p.line.carry + (static_cast<long>(line()) * 128 + half * 64) * 128 + (warp & 3) * 32 + lane
                   : p.state + ((static_cast<long>(p.state_slot[e]) * p.heads + h) * p.D + half * 64) * p.Dv + cb0 + (warp & 3) * 32 + lane;
          if (out) step = 128;
        }
        asm volatile("" : "+l"(gS), "+l"(step));             // the addresses are not kept from the load to here: 128 registers
#pragma unroll
        for (int d = 0; d < 64; ++d, gS += step)
          if (d < rows) *gS = S[d];
        if (out) {
          __threadfence();
          named_barrier_sync(2, NH * 128);
          if (threadIdx.x == 4 * 32) asm volatile("st.release.gpu.global.b32 [%0], 1;" ::"l"(p.line.handed + line()) : "memory");
        }
      } else {
        for (int n = 0; n < n_chunks; ++n) {
          for (int c = 0; c < 4; ++c) mbar_arrive(&sp_full[c]);
          mbar_wait_quiet(&kq_full[n & 1], (n >> 1) & 1);
          mbar_arrive(&sc_free[n & 1]);
          mbar_wait_quiet(ds_full, n & 1);
        }
      }
    }
  } else if (warp < 16) {
    // ============================== terms of k and q ==============================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    const int tid = threadIdx.x - 12 * 32;
    // a row (token of K or Q) per group of DP / 16 threads, 16 values in two runs of eight a thread; RW rows at a time
    constexpr int TR = DP / 16, RW = 128 / TR, NR = 2 * kC / RW;
    const int d0 = (tid % TR) * 8, r0 = tid / TR;
    float beta, gd;
    auto fetch_sc = [&](int t) {
      beta = 0.f;
      gd = 1.f;
      if (tid < kC && t + tid < t1) {
        if (DELTA) beta = p.beta[static_cast<long>(t + tid) * p.heads + h];
        gd = p.decay[static_cast<long>(t + tid) * p.heads + h];
      }
    };
#pragma unroll 1
    for (int i = first; i < last; ++i, turn()) {
      if (LINE) take(i);
      fetch_sc(t0);
      for (int n = 0; n < n_chunks; ++n) {
        const int st = n & 1, t = t0 + n * kC;
        const uint32_t ph2 = (n >> 1) & 1;
        float2 c = make_float2(gd, 0.f), w = make_float2(1.f, 0.f);      // g_1 .. g_i and g_{i+1} .. g_n
        if (warp == 12) {
          w.x = __shfl_down_sync(0xffffffffu, gd, 1);
          if (lane == 31) w.x = 1.f;
#pragma unroll 1
          for (int m = 1; m < 32; m <<= 1) {
            const float2 a = make_float2(__shfl_up_sync(0xffffffffu, c.x, m), __shfl_up_sync(0xffffffffu, c.y, m));
            const float2 b = make_float2(__shfl_down_sync(0xffffffffu, w.x, m), __shfl_down_sync(0xffffffffu, w.y, m));
            if (lane >= m) c = mul_wide(c, a);
            if (lane + m < 32) w = mul_wide(w, b);
          }
        }
        mbar_wait_quiet(&kq_free[st], ph2 ^ 1);
        mbar_wait_quiet(&sc_free[st], ph2 ^ 1);
        if (warp == 12) {
          float* sc = reinterpret_cast<float*>(smem + L::kSc + st * L::kScStage);
          sc[lane] = beta;
          sc[kC + lane] = c.x + c.y;
          sc[2 * kC + lane] = w.x + w.y;
          sc[3 * kC + lane] = gd;
          sc[4 * kC + lane] = 1.f;
        }
        fetch_sc(t + kC);
        mbar_wait_quiet(&raw_full[st], ph2);
        uint8_t* tile = smem + L::kKQ + st * L::kKQStage;
        const float* raw = reinterpret_cast<const float*>(smem + L::kRaw + st * L::kRawStage);
#pragma unroll 1
        for (int s = 0; s < NR; ++s)
#pragma unroll 1
          for (int q = 0; q < 2; ++q) {
            const int row = s * RW + r0, d = d0 + q * (DP / 2), chunk = (d & 63) >> 3;
            const float4 a = *reinterpret_cast<const float4*>(raw + row * DP + d), b = *reinterpret_cast<const float4*>(raw + row * DP + d + 4);
            uint32_t y[3][4];
            split3(a.x, a.y, y[0][0], y[1][0], y[2][0]);
            split3(a.z, a.w, y[0][1], y[1][1], y[2][1]);
            split3(b.x, b.y, y[0][2], y[1][2], y[2][2]);
            split3(b.z, b.w, y[0][3], y[1][3], y[2][3]);
#pragma unroll
            for (int m = 0; m < 3; ++m)
              *reinterpret_cast<uint4*>(tile + (m * NH + (d >> 6)) * kDcTile + row * 128 + ((chunk ^ (row & 7)) << 4)) =
                  make_uint4(y[m][0], y[m][1], y[m][2], y[m][3]);
          }
        mbar_arrive(&raw_free[st]);
        fence_proxy_async_smem();
        mbar_arrive(&kq_full[st]);
      }
    }
  } else if (warp < 20) {
    // ============================== Gram matrices ==============================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    // rows of this thread: those of a 64-row accumulator are sixteen lanes of each warp's quarter
    const int gi = ((warp & 3) * 16 + (lane & 15)) & (kC - 1);
    const bool is_q = (warp & 3) >= 2, have = lane < 16;
#pragma unroll 1
    for (int i = first; i < last; ++i, turn()) {
      if (LINE) take(i);
      for (int n = 0; n < n_chunks; ++n) {
        const int st = n & 1;
        const uint32_t ph2 = (n >> 1) & 1;
        mbar_wait_quiet(&kq_full[st], ph2);
        mbar_wait_quiet(&kq_free[st], ph2 ^ 1);                      // the products that read the stage's Gram matrices
        const float* sc = reinterpret_cast<const float*>(smem + L::kSc + st * L::kScStage);
        const float bi = is_q ? 1.f : sc[gi];
        float2 w = make_float2(1.f, 0.f);                    // G(gi, j)
        mbar_wait_quiet(gram_full, n & 1);
        tc_fence_after();
        uint8_t* mt = smem + L::kM + st * L::kMStage;
        float* lj = reinterpret_cast<float*>(smem + L::kL + st * L::kLStage);
#pragma unroll 1
        for (int c = kC - 8; c >= 0; c -= 8) {
          uint32_t ga[8], gb[8];
          tmem_ld_32x32b_x8(tmem + Tm::kG1 + c + lane_off, ga);
          tmem_ld_32x32b_x8(tmem + Tm::kG2 + c + lane_off, gb);
          float m[8];
#pragma unroll
          for (int a = 7; a >= 0; --a) {
            const int j = c + a;
            const float gj = j < gi ? sc[3 * kC + j + 1] : 1.f;
            w = mul_wide(w, make_float2(gj, 0.f));
            m[a] = bi * (w.x + w.y);
          }
          tmem_ld_wait();
#pragma unroll
          for (int a = 0; a < 8; ++a)
            m[a] = c + a < gi || (is_q && c + a == gi) ? m[a] * (__uint_as_float(ga[a]) + __uint_as_float(gb[a])) : 0.f;
          if (have && is_q) {
            uint32_t y[3][4];
#pragma unroll
            for (int a = 0; a < 8; a += 2) split3(m[a], m[a + 1], y[0][a / 2], y[1][a / 2], y[2][a / 2]);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
              const int chunk = (b == 1 ? 4 : 0) + c / 8;
              *reinterpret_cast<uint4*>(mt + (b == 2 ? kC * 128 : 0) + gi * 128 + ((chunk ^ (gi & 7)) << 4)) =
                  make_uint4(y[b][0], y[b][1], y[b][2], y[b][3]);
            }
          } else if (have && DELTA) {
#pragma unroll
            for (int a = 0; a < 8; ++a) lj[(c + a) * kC + gi] = m[a];
          }
        }
        tc_fence_before();
        mbar_arrive(gram_free);
        mbar_arrive(&sc_free[st]);
        fence_proxy_async_smem();
        mbar_arrive(&lm_full[st]);
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp > 20) {
      // ============================== q, k and v ==============================
      const int tid = threadIdx.x - 21 * 32;
      if (WIDE) {
        float* all = reinterpret_cast<float*>(smem + L::kRaw);
        if (p.D < DP || p.Dv % 128 != 0)                    // columns that no copy reaches
          for (int x = tid; x < 2 * L::kRawStage / 4; x += kDcLoaders) all[x] = 0.f;
        fence_proxy_async_smem();                           // the zeros lie under what the copies bring: in front of them for the asynchronous proxy too
        named_barrier_sync(1, kDcLoaders);
      }
#pragma unroll 1
      for (int i = first; i < last; ++i, turn()) {
        if (LINE) take(i);
        const float* src = p.qkv + static_cast<long>(h / (p.heads / p.kv_heads)) * p.D;
        const float* vsrc = p.qkv + p.col_v + static_cast<long>(h) * p.Dv + cb0;
        const int vcols = min(p.Dv - cb0, 128);
        for (int n = 0; n < n_chunks && (!WIDE || warp == 21); ++n) {
          const int st = n & 1, t = t0 + n * kC;
          mbar_wait_quiet(&raw_free[st], ((n >> 1) & 1) ^ 1);
          float* raw = reinterpret_cast<float*>(smem + L::kRaw + st * L::kRawStage);
          float* rv = reinterpret_cast<float*>(smem + L::kRaw + st * L::kRawStage + L::kRawV);
          if (WIDE) {                                         // a lane per token
            if (t + lane < t1) {
              const long row = static_cast<long>(t + lane) * p.sq;
              mbar_arrive_expect_tx(&raw_full[st], (2 * p.D + vcols) * 4);
              bulk_load(raw + lane * DP, src + p.col_k + row, p.D * 4, &raw_full[st]);
              bulk_load(raw + (kC + lane) * DP, src + row, p.D * 4, &raw_full[st]);
              bulk_load(rv + lane * 128, vsrc + row, vcols * 4, &raw_full[st]);
            } else {
              for (int d = 0; d < DP; d += 4) {
                *reinterpret_cast<float4*>(raw + lane * DP + d) = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(raw + (kC + lane) * DP + d) = make_float4(0.f, 0.f, 0.f, 0.f);
              }
              for (int c = 0; c < 128; c += 4) *reinterpret_cast<float4*>(rv + lane * 128 + c) = make_float4(0.f, 0.f, 0.f, 0.f);
              mbar_arrive(&raw_full[st]);
            }
          } else {
#pragma unroll 1
            for (int x = tid; x < 2 * kC * DP; x += kDcLoaders) {              // rows 0..31 are K, 32..63 Q
              const int row = x / DP, d = x % DP, i = row & (kC - 1);
              const bool ok = t + i < t1 && d < p.D;
              cp_async_zfill(raw + row * DP + d, ok ? src + static_cast<long>(t + i) * p.sq + (row < kC ? p.col_k : 0) + d : p.qkv, ok);
            }
#pragma unroll 1
            for (int x = tid; x < kC * 128; x += kDcLoaders) {
              const int i = x / 128, c = x % 128;
              const bool ok = t + i < t1 && c < vcols;
              cp_async_zfill(rv + i * 128 + c, ok ? vsrc + static_cast<long>(t + i) * p.sq + c : p.qkv, ok);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&raw_full[st])) : "memory");
          }
        }
      }
    } else {
      // ============================== MMA issuer ==============================
      // the whole warp runs the loops, one lane issues: what is the same in all lanes stays in uniform registers
      const uint32_t leader = elect_one(), tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
      constexpr uint32_t id_gram = make_idesc(2 * kC, kC, 1, 1), id_rq = make_idesc(128, kC, 1, 1);
      constexpr uint32_t id_ds = make_idesc_bmn(128, 64), id_o2 = make_idesc(128, kC, 1, 1);
      // descriptors of the first tiles; what is added is in units of 16 bytes
      const uint64_t kq0 = make_smem_desc_sw128(smem_u32(smem + L::kKQ)), kt0 = make_smem_desc_sw128_mn(smem_u32(smem + L::kKQ), kDcTile);
      const uint64_t m0 = make_smem_desc_sw128(smem_u32(smem + L::kM));
      constexpr int kTerm = NH * kDcTile / 16, kHalfTile = kDcTile / 16, kStep = 2;       // to the next term, half, 16 columns
      auto gram = [&](int n) {
        const int st = n & 1;
        const uint64_t d = kq0 + st * (L::kKQStage / 16);
        mbar_wait_quiet(&kq_full[st], (n >> 1) & 1);
        if (n > 0) mbar_wait_quiet(gram_free, (n - 1) & 1);
        tc_fence_after();
#pragma unroll 1
        for (int pr = 0; pr < 6; ++pr) {
          const uint64_t a = d + pair_a(pr) * kTerm, b = d + pair_b(pr) * kTerm;
#pragma unroll
          for (int k = 0; k < 4 * NH; ++k) {
            const int off = (k >> 2) * kHalfTile + (k & 3) * kStep;
            dc_mma(leader, tmem_u + (pr == 5 && k >= 2 * NH ? Tm::kG2 : Tm::kG1), a + off, b + off, id_gram, (pr == 0 && k == 0) || (pr == 5 && k == 2 * NH) ? 0u : 1u);
          }
        }
        dc_commit(leader, gram_full);
      };
#pragma unroll 1
      for (int i = first; i < last; ++i, turn()) {
        if (LINE) take(i);
        if (n_chunks > 0) gram(0);
#pragma unroll 1
        for (int n = 0; n < n_chunks; ++n) {
          const int st = n & 1;
          const uint64_t d = kq0 + st * (L::kKQStage / 16), dt = kt0 + st * (L::kKQStage / 16), dm = m0 + st * (L::kMStage / 16);
          auto rq = [&](int pr, int k, int kq, bool second, bool first) {      // kq: 0 K, 1 Q, 32 rows further and 32 columns
            dc_mma_ts(leader, tmem_u + (second ? Tm::kR2 : Tm::kR1) + kq * kC, tmem_u + Tm::kHalf * (k >> 2) + 32 * pair_a(pr) + 8 * (k & 3),
                        d + pair_b(pr) * kTerm + (k >> 2) * kHalfTile + (k & 3) * kStep + kq * (kC * 8), id_rq, first ? 0u : 1u);
          };
          // K, which the solve waits for: the small pairs as the terms come
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            mbar_wait_quiet(&sp_full[c], n & 1);
            tc_fence_after();
#pragma unroll
            for (int pr = 0; pr < 5; ++pr)
#pragma unroll
              for (int hf = 0; hf < NH; ++hf) rq(pr, 4 * hf + c, 0, false, c == 0 && pr == 0 && hf == 0);
          }
#pragma unroll
          for (int k = 0; k < 4 * NH; ++k) rq(5, k, 0, k >= 2 * NH, k == 2 * NH);
          dc_commit(leader, rk_full);
#pragma unroll 1
          for (int pr = 0; pr < 6; ++pr)
#pragma unroll
            for (int k = 0; k < 4 * NH; ++k) rq(pr, k, 1, pr == 5 && k >= 2 * NH, (pr == 0 && k == 0) || (pr == 5 && k == 2 * NH));
          dc_commit(leader, rq_full);
          if (n + 1 < n_chunks) gram(n + 1);
          mbar_wait_quiet(uh_full, n & 1);
          tc_fence_after();
#pragma unroll
          for (int hf = 0; hf < NH; ++hf)
#pragma unroll
            for (int pr = 0; pr < 6; ++pr)
#pragma unroll
              for (int k = 0; k < kC / 16; ++k)               // 16 tokens: 16 rows of 128 bytes
                dc_mma_ts(leader, tmem_u + Tm::kHalf * hf, tmem_u + Tm::uh(pair_a(pr)) + 8 * k, dt + pair_b(pr) * kTerm + hf * kHalfTile + k * 128, id_ds,
                            pr == 0 && k == 0 ? 0u : 1u);
          dc_commit(leader, ds_full);
          mbar_wait_quiet(u_full, n & 1);
          mbar_wait_quiet(&lm_full[st], (n >> 1) & 1);
          tc_fence_after();
#pragma unroll 1
          for (int pr = 0; pr < 6; ++pr)
#pragma unroll
            for (int k = 0; k < kC / 16; ++k)                 // terms 0 and 1 side by side, 2 in a tile of its own
              dc_mma_ts(leader, tmem_u + Tm::kO2, tmem_u + Tm::kU + 16 * pair_a(pr) + 8 * k,
                          dm + (pair_b(pr) == 2 ? kC * 128 / 16 : pair_b(pr) * 4) + k * kStep, id_o2, pr == 0 && k == 0 ? 0u : 1u);
          dc_commit(leader, o2_full);
          dc_commit(leader, &kq_free[st]);
        }
        // nothing that is still under way arrives at a barrier that starts anew
        if (LINE)
          for (int n = max(0, n_chunks - 2); n < n_chunks; ++n) mbar_wait_quiet(&kq_free[n & 1], (n >> 1) & 1);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 20) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int DP, bool DELTA, bool WIDE, bool LINE>
cudaError_t launch_delta_chunk(unsigned grid, const DcParams& p, cudaStream_t s) {
  auto kern = delta_chunk_tc_kernel<DP, DELTA, WIDE, LINE>;
  constexpr int smem = DcSmem<DP>::kTotal;
  static const cudaError_t configured = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (configured != cudaSuccess) return configured;
  kern<<<grid, kDcThreads, smem, s>>>(p);
  return cudaGetLastError();
}

}  // namespace
}  // namespace nrl

// D <= 128, one decay per head; beta == nullptr: plain accumulation; rows16: rows of q, k and v start and end on 16-byte boundaries; line: null, or (rows16)
// nrl_delta_line_bytes() of scratch with which `blocks` blocks share the chunks of all items, where that pays or it is forced
extern "C" long nrl_delta_line_bytes(long E, int heads, int Dv, int blocks) {
  return blocks * (128l * 128 * 4 + 12) + 16 + (E * heads * ((Dv + 127) / 128) + blocks) * static_cast<long>(sizeof(nrl::DcSegment));
}
static nrl::DcLine line_in(void* scratch, int blocks) {
  nrl::DcLine l{};
  l.carry = static_cast<float*>(scratch);
  l.first = reinterpret_cast<int*>(l.carry + blocks * 128l * 128);
  l.last = l.first + blocks;
  l.handed = l.last + blocks;
  l.taken = l.handed + blocks;
  l.ticket = l.taken + 1;
  l.segments = reinterpret_cast<nrl::DcSegment*>(l.taken + 4);
  return l;
}
extern "C" int nrl_delta_line_pays(const long* tokens, long E, int heads, int Dv, int blocks) {
  const long items = static_cast<long>(heads) * ((Dv + 127) / 128);
  std::vector<long> n(E);
  long total = 0;
  for (long e = 0; e < E; ++e) total += n[e] = std::max(1l, (tokens[e] + nrl::kC - 1) / nrl::kC);
  std::sort(n.begin(), n.end(), std::greater<long>());
  const long share = (total * items + blocks - 1) / blocks;
  long whole = share;
  for (long e = 0; e < E; ++e) whole = std::max(whole, ((e + 1) * items + blocks - 1) / blocks * n[e]);
  return E > 0 && nrl::line_pays(std::max(n[0], share), whole);
}
extern "C" cudaError_t nrl_delta_line(const int* cu, int E, int heads, int Dv, bool forced, void* line, int blocks, cudaStream_t s) {
  if (E > nrl::kDcMaxEntries) return cudaErrorInvalidValue;
  nrl::delta_line_kernel<<<1, 1024, 0, s>>>(cu, E, heads, (Dv + 127) / 128, blocks, forced, line_in(line, blocks));
  return cudaGetLastError();
}
extern "C" cudaError_t nrl_delta_chunk_tc(const float* qkv, long sq, int col_k, int col_v, const float* beta, const float* decay, float* state, float* o,
                                          const int* cu, const int* start, const int* state_slot, int E, int heads, int kv_heads, int D, int Dv,
                                          bool rows16, void* line, int blocks, bool forced, cudaStream_t s) {
  nrl::DcParams p{qkv, beta, decay, state, o, cu, start, state_slot, sq, col_k, col_v, heads, kv_heads, D, Dv, {}};
  const int parts = (Dv + 127) / 128;
  const unsigned grid = static_cast<unsigned>(E) * heads * parts;
  if (line != nullptr) {
    if (!rows16) return cudaErrorInvalidValue;
    p.line = line_in(line, blocks);
    if (const cudaError_t e = nrl_delta_line(cu, E, heads, Dv, forced, line, blocks, s); e != cudaSuccess) return e;
  }
#define NRL_DC(P_, B_)                                                 \
  if ((D <= 64 ? 64 : 128) == P_ && (beta != nullptr) == B_) {           \
    if (line != nullptr) {                                               \
      const cudaError_t e = nrl::launch_delta_chunk<P_, B_, true, true>(static_cast<unsigned>(blocks), p, s);       \
      if (e != cudaSuccess || forced) return e;                          \
    }                                                                    \
    return (rows16 ? nrl::launch_delta_chunk<P_, B_, true, false> : nrl::launch_delta_chunk<P_, B_, false, false>)(grid, p, s); \
  }
  NRL_DC(64, true) NRL_DC(64, false) NRL_DC(128, true) NRL_DC(128, false)
#undef NRL_DC
  return cudaErrorInvalidValue;
}
