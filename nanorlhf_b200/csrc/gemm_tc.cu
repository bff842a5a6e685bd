// gemm_tc: the general tcgen05 / TMEM / TMA GEMM of the training, log-prob and reward paths (hand-written PTX).
//
//   D[M,N] = alpha * ( opA(A) . opB(B)^T  +  A2 . B2^T )  (+ bias[N]) (GELU)          bf16 in, fp32 accumulate
//
// One kernel template covers what the reference gets from cuBLAS behind every nn.Linear / peft LoRA layer / torch.bmm
// (GRPO/grpo_trainer.py:543-556,652-660; GRPO/grpo.py:189-192,228-243):
//
//   * CG = 1 | 2      cta_group::1 (one CTA, 128 x BN tile) or cta_group::2 (a CTA pair of one TPC computes a 256 x BN
//                     tile; each CTA TMA-loads its own 128 rows of A and only HALF of the B tile, one elected thread of
//                     the leader CTA issues `tcgen05.mma.cta_group::2`, commits are multicast to both CTAs' barriers).
//                     Per k-block an SM ingests 16 KB + BN*64 B instead of 16 KB + BN*128 B: the L2->SM stream and the
//                     smem operand reads -- what bounds the 1-CTA kernel -- drop by a third (measured: 1.15-1.25x).
//   * BN = 64 | 128 | 192 | 256   picked on the host by wave efficiency (N = 1536 outputs: 192 fills 2.9 of 3 waves
//                     where 256 fills 2.2 of 3).
//   * A_MN / B_MN     either operand may be "MN-major" (the contraction index is the ROW of the stored matrix).  That is
//                     what makes dgrad ( dX = dY . W : B = W[N,K] read as [k=N rows][n=K cols] ) and wgrad
//                     ( dW = dY^T . X : both operands token-major ) run on the same kernel with NO transposed copies:
//                     TMA lands [64 k-rows x 64 mn-cols] panels and the UMMA descriptor addresses them as MN-major.
//   * dual source K   a second operand pair (A2, B2) contributes K2 further contraction columns into the same TMEM
//                     accumulator: LoRA  y = x W^T + (s x A^T) B^T  is ONE GEMM with K + r columns instead of a base
//                     GEMM, an adapter GEMM and an add pass over [M,N]; likewise dX = dY W + (s dY B) A.
//   * epilogues       EPI_BF16: alpha, bias, exact GELU -> bf16 through swizzled smem + TMA store;
//                     EPI_F32 : fp32 row-major out (+)= alpha * acc  (weight-gradient accumulation, lm-head dW).
//
// Pipeline (per CTA, 320 threads): warp 0 = TMA producer, warp 1 = MMA issuer (+ TMEM allocator), warps 2-9 = epilogue;
// smem ring of kStages k-blocks behind full/empty mbarriers, two TMEM accumulators so the epilogue of tile i overlaps the
// main loop of tile i+1, persistent grid with a grouped (L2-friendly) tile order.
// An epilogue warp owns 32 rows of every other 64-column chunk and stages and stores them on its own (4 KB slab, one TMA store), so no
// barrier joins the warps.  With four warps that met at two barriers per chunk and read the bias value by value, a 128 x 256 tile's
// epilogue took longer than a main loop of K = 1024: the six linears of a reward layer (24 571 tokens) 742 -> 429 us, its bias tables
// (K = 64) 235 -> 92 us each; nothing changes above K = 4096.
#include "cluster_read.h"
#include "common.cuh"
#include "gemm_tc.h"
#include "launch.h"
#include "per_device.h"

namespace nrl {
namespace tc {

constexpr int BLOCK_M = 128;        // rows per CTA (a CTA pair covers 256)
constexpr int BLOCK_K = 64;         // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int kEpiWarps = 8;        // two per TMEM lane quadrant
constexpr int kEpiThreads = 32 * kEpiWarps;
constexpr int kThreads = 64 + kEpiThreads;
constexpr int kABytes = BLOCK_M * BLOCK_K * 2;      // 16 KB
constexpr int kPanelBytes = 64 * 128;               // one [64 x 64] bf16 panel of an MN-major operand
constexpr int kSlabBytes = 32 * 128;                // 32 rows x 64 bf16 output slab of an epilogue warp
constexpr int kStagingBytes = kEpiWarps * kSlabBytes;
constexpr int kSmemBudget = 227 * 1024;
constexpr uint32_t kPeerMask = 0xFEFFFFFFu;         // clears the CTA-pair peer bit of a shared::cluster address
constexpr int GROUP_M = 8;                          // tile rows per L2 super-row
constexpr int kMaxClusterSplits = 8;                // blocks of a portable cluster

template <int CG, int BN, bool B_MN = false, int SLABS = 1>      // SLABS: output slabs of an epilogue warp
struct Cfg {
  static constexpr int kBRows = BN / CG;                                  // B rows (n) this CTA contributes per k-block
  // an MN-major B tile is made of whole [64 k x 64 n] panels: 96 columns (BN = 192 on a CTA pair) load two panels, the
  // MMA reads the first 96 columns of them (the surplus 32 belong to the peer / the next tile and are ignored)
  static constexpr int kBPanels = (kBRows + 63) / 64;
  static constexpr int kBBytes = B_MN ? kBPanels * kPanelBytes : kBRows * BLOCK_K * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStaging = SLABS * kStagingBytes;
  static constexpr int kStagesFit = (kSmemBudget - kStaging - 1024) / kStageBytes;
  static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;
  static constexpr int kStagingOff = kStages * kStageBytes;
  static constexpr int kBarOff = kStagingOff + kStaging;
  static constexpr int kTotal = kBarOff + 512;
  static constexpr uint32_t kTmemCols = (2 * BN <= 128) ? 128 : (2 * BN <= 256) ? 256 : 512;
  static_assert(kStageBytes % 1024 == 0, "stages must keep the 1024-byte swizzle alignment");
};

NRL_DEVICE uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
NRL_DEVICE void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int CG>
NRL_DEVICE void tmem_alloc_cg(uint32_t* smem_dst, uint32_t ncols) {
  if (CG == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
}
template <int CG>
NRL_DEVICE void tmem_dealloc_cg(uint32_t taddr, uint32_t ncols) {
  if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
template <int CG>
NRL_DEVICE void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if (CG == 1) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  }
}
template <int CG>
NRL_DEVICE void umma_fp8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if (CG == 1) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  }
}
// all MMAs issued so far by this thread arrive on `bar` when they retire (CG = 2: on the barrier at the same offset in
// BOTH CTAs of the pair)
// (`pair`: the two blocks' bits among the cluster's)
template <int CG>
NRL_DEVICE void umma_commit_cg(uint64_t* bar, uint32_t pair = 3) {
  if (CG == 1) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
  } else {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(pair)) : "memory");
  }
}
// TMA tile load; CG = 2: the transaction bytes are credited to the LEADER CTA's barrier (peer bit cleared)
template <int CG>
NRL_DEVICE void tma_load_cg(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1) {
  if (CG == 1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1) : "memory");
  } else {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar) & kPeerMask), "r"(c0), "r"(c1) : "memory");
  }
}
NRL_DEVICE void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & kPeerMask) : "memory");
}
NRL_DEVICE constexpr uint32_t make_idesc_tc(uint32_t M, uint32_t N, bool a_mn, bool b_mn) {     // bf16 x bf16 -> fp32
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((N >> 3) << 17) |
         ((M >> 4) << 24);
}

NRL_DEVICE float gelu_erf_tc(float x) {          // Abramowitz-Stegun 7.1.26, |err| < 1.5e-7 (see gemm_sm100.cu)
  const float z = fabsf(x) * 0.70710678118654752f;
  const float t = __fdividef(1.f, fmaf(0.3275911f, z, 1.f));
  float poly = fmaf(1.061405429f, t, -1.453152027f);
  poly = fmaf(poly, t, 1.421413741f);
  poly = fmaf(poly, t, -0.284496736f);
  poly = fmaf(poly, t, 0.254829592f);
  const float erf_abs = 1.f - poly * t * exp2f(-z * z * 1.4426950408889634f);
  return 0.5f * x * (1.f + copysignf(erf_abs, x));
}

struct TileCoord {
  int m_tile, n_blk;          // m_tile in units of CG*128 rows
};
NRL_DEVICE TileCoord tile_coord(int t, int num_m, int num_n) {
  const int per_group = GROUP_M * num_n;
  const int g = t / per_group, r = t - g * per_group;
  const int gsz = min(GROUP_M, num_m - g * GROUP_M);
  TileCoord c;
  c.n_blk = r / gsz;
  c.m_tile = g * GROUP_M + (r - c.n_blk * gsz);
  return c;
}

template <int CG>
NRL_DEVICE void tma_load3_cg(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2) {
  if (CG == 1) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
  } else {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar) & kPeerMask), "r"(c0), "r"(c1), "r"(c2) : "memory");
  }
}
NRL_DEVICE void tma_store_3d(const CUtensorMap* m, const void* smem_src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

// 32 rows of W words, one row per lane, handed out in pieces of 16 bytes so that W / 4 neighbouring lanes hold neighbouring pieces of a row:
// put(step, row, piece, words).  The plain stores of the float and grouped epilogues go through it: a lane per row wrote 16 bytes into each of 32
// lines at a time, which eight warps at once took longer for than four (4096 x 1536 -> 151 936
// floats 1699 us, with eight 1893, handed out 1469; added to 3552, 1590; 16 384 tokens over 64 experts 721, 900, 563).
template <int W, class F>
NRL_DEVICE void warp_rows_out(uint8_t* slab, const uint32_t (&w)[W], int lane, F&& put) {
  constexpr int P = W / 4;
  __syncwarp();                                           // the slab's last rows have been read
#pragma unroll
  for (int q = 0; q < P; ++q)
    *reinterpret_cast<uint4*>(slab + lane * (W * 4) + ((q ^ (lane & (P - 1))) * 16)) = make_uint4(w[q * 4], w[q * 4 + 1], w[q * 4 + 2], w[q * 4 + 3]);
  __syncwarp();
  const int q = lane % P;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int r = i * (32 / P) + lane / P;
    put(i, r, q, *reinterpret_cast<const uint4*>(slab + r * (W * 4) + ((q ^ (r & (P - 1))) * 16)));
  }
}

// FP8: A and B are e4m3 bytes, K-major (a 128-byte swizzle row = 128 contraction elements), the MMA is kind::f8f6f4
// (K = 32 per instruction, twice the bf16 rate) and the epilogue applies the per-row (token) and per-column (output
// channel) dequantisation scales -- the sampler's fp8 rollout GEMMs.
// PAIR (CTA pairs, BN = 256): act = silu(x Wg^T) * (x Wu^T) from two separate weights.  The leader loads 128 rows of the gate's
// weight, its peer the same 128 rows of the up weight, so the accumulator's halves are gate and up of the same features; the adapters'
// columns follow (first the gate's, then the up's), each weight taking zeros (rows behind its end) for the other's.
template <int CG, int BN, bool A_MN, bool B_MN, int EPI, bool SPLIT = false, bool BATCH = false, bool FP8 = false, bool GROUPED = false,
          bool PAIR = false, bool CLUSTER = false, bool SUM = false, bool CAT = false, bool MULTI = false>
NRL_DEVICE void gemm_tc_body(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmA2, const CUtensorMap& tmB2,
                             const CUtensorMap& tmD, const TcParams& p, const CUtensorMap* more = nullptr, int unit0 = 0, const TcCat* cat = nullptr) {
  // more: PAIR the up adapter's columns, then (EPI_SWIGLU_KEEP) gate and up; EPI_DSWIGLU gate, up, d up; SUM kSumPairs maps of A and as many of B;
  // CAT kCatMax each of B, A2, B2, D
  using C = Cfg<CG, BN, B_MN, EPI == EPI_DSWIGLU ? 2 : 1>;
  constexpr bool kPlainStores = EPI == EPI_F32 || EPI == EPI_LOGPROB || EPI == EPI_GRP_SWIGLU || EPI == EPI_GRP_RELU2;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + C::kBarOff);      // CG = 2: the leader's are the live ones
  uint64_t* empty_bar = full_bar + C::kStages;                              // per CTA (multicast commit)
  uint64_t* tmem_full = empty_bar + C::kStages;                             // [2] per CTA (multicast commit)
  uint64_t* tmem_empty = tmem_full + 2;                                     // [2] CG = 2: the leader's are the live ones
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = (CG == 2) ? cluster_ctarank() & 1u : 0u;
  const uint32_t pair = (CG == 2 && CLUSTER) ? 3u << (cluster_ctarank() & ~1u) : 3u;
  const bool leader = rank == 0;
  const int num_m = (p.M + CG * BLOCK_M - 1) / (CG * BLOCK_M);
  const int num_n = CAT ? cat->end[kCatMax - 1] : (p.N + BN - 1) / BN;
  constexpr int kElemsPerKB = FP8 ? 2 * BLOCK_K : BLOCK_K;                  // 128 bytes of contraction per k-block either way
  const int num_kb1 = (p.K + kElemsPerKB - 1) / kElemsPerKB;
  const int num_kb2 = (p.K2 + kElemsPerKB - 1) / kElemsPerKB;
  const int num_kb = SUM ? p.sum_end[kSumPairs - 1] : num_kb1 + (PAIR ? 2 : 1) * num_kb2;
  const int splits = SPLIT ? p.splits : 1;
  const int kb_per_split = (num_kb + splits - 1) / splits;
  const int tiles_per_batch = num_m * num_n;
  const int unit = blockIdx.x / CG - unit0, num_units = gridDim.x / CG;      // unit0: blocks that work on other products
  volatile int* s_last = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  if (warp == 0 && lane == 0) {
    if (SUM)
      for (int i = 0; i < 2 * kSumPairs; ++i) tma_prefetch_desc(more + i);
    else tma_prefetch_desc(&tmA);
    if (CAT)
      for (int i = 0; i < 4 * kCatMax; ++i) tma_prefetch_desc(more + i);
    if (!SUM && !CAT) tma_prefetch_desc(&tmB);
    if (!SUM && !CAT && p.K2 > 0) {
      tma_prefetch_desc(&tmA2);
      tma_prefetch_desc(&tmB2);
    }
    if (!kPlainStores && !CAT) tma_prefetch_desc(&tmD);
  }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < C::kStages; ++i) {
      mbar_init(&full_bar[i], 1);                       // the (leader's) producer thread + the transaction bytes
      mbar_init(&empty_bar[i], 1);                      // one (multicast) commit
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);                      // one (multicast) commit
      mbar_init(&tmem_empty[i], CG * kEpiWarps); // the epilogue warps (of both CTAs)
    }
    if (EPI == EPI_DSWIGLU)
      for (int i = 0; i < kEpiWarps; ++i) mbar_init(reinterpret_cast<uint64_t*>(smem + C::kBarOff + 256) + i, 1);
    fence_mbar_init();
  }
  if (CG == 2) cluster_sync_all();                      // the peer's barriers exist before anything remote is signalled
  if (warp == 1) {
    __syncwarp();
    tmem_alloc_cg<CG>(tmem_ptr, C::kTmemCols);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  pdl_wait();
  pdl_launch_dependents();
  // SPLIT: work item = (tile, k-range), splits of a tile adjacent.  BATCH: work item = (batch, tile), third TMA coordinate
  // GROUPED: work item = (row tile of the device-side table, column block); the column blocks of a row tile are adjacent
  // EPI_LOGPROB: work item = (row tile, range of column tiles), row tiles varying fastest: blocks that share a range walk its weight together
  constexpr bool kRanges = EPI == EPI_LOGPROB;
  const int n_per_range = kRanges ? (num_n + p.col_ranges - 1) / p.col_ranges : 1;
  auto range_of = [&](int w, TileCoord& c) {               // first column tile in c, returns the end
    if (!kRanges) return c.n_blk + 1;
    const int g = w / num_m;
    c.m_tile = w - g * num_m;
    c.n_blk = g * n_per_range;
    return min(num_n, c.n_blk + n_per_range);
  };
  auto product_of = [&](int& n_blk) {                      // CAT: the product of a column tile, which becomes one of that product
    int i = 0;
    while (n_blk >= cat->end[i]) ++i;                      // n_blk < end[kCatMax - 1]
    if (i > 0) n_blk -= cat->end[i - 1];
    return i;
  };
  const int num_work = GROUPED ? __ldg(p.grp_num_tiles) * num_n : kRanges ? num_m * p.col_ranges : tiles_per_batch * (BATCH ? p.batch : splits);

  if (warp == 0) {
    // ================================ TMA producer (every CTA) ================================
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int w = unit; w < num_work; w += num_units) {
        const int bidx = BATCH ? w / tiles_per_batch : 0;
        TileCoord c = GROUPED || kRanges ? TileCoord{0, 0} : tile_coord(BATCH ? w % tiles_per_batch : w / splits, num_m, num_n);
        const int n_end = range_of(w, c);
        for (; c.n_blk < n_end; ++c.n_blk) {
          int m0 = (c.m_tile * CG + static_cast<int>(rank)) * BLOCK_M;
          int n0 = c.n_blk * BN + static_cast<int>(rank) * C::kBRows;
          if (GROUPED) {
            const int mt = w / num_n;
            c.n_blk = w - mt * num_n;
            m0 = __ldg(p.grp_tiles + 3 * mt + 1);
            n0 = __ldg(p.grp_tiles + 3 * mt) * p.N + c.n_blk * BN;      // the expert's block of B rows
          }
          if (PAIR) n0 = c.n_blk * (BN / 2);
          int which = 0;
          if (CAT) {
            int blk = c.n_blk;
            which = product_of(blk);
            n0 = blk * BN + static_cast<int>(rank) * C::kBRows;
          }
          const int kb_lo = BATCH ? 0 : (w % splits) * kb_per_split, kb_hi = BATCH ? num_kb : min(num_kb, kb_lo + kb_per_split);
          for (int kb = kb_lo; kb < kb_hi; ++kb) {
            mbar_wait(&empty_bar[stage], phase ^ 1);
            uint8_t* sa = smem + stage * C::kStageBytes;
            uint8_t* sb = sa + kABytes;
            if (leader) mbar_arrive_expect_tx(&full_bar[stage], CG * C::kStageBytes);
            const bool second = kb >= num_kb1;
            const CUtensorMap* ma = second ? &tmA2 : &tmA;
            const CUtensorMap* mb = second ? &tmB2 : &tmB;
            int k0 = (second ? kb - num_kb1 : kb) * kElemsPerKB;
            if (CAT) {
              if (second) ma = more + kCatMax + which;
              mb = more + (second ? 2 * kCatMax : 0) + which;
            }
            if (SUM) {
              int i = 0;
              while (kb >= p.sum_end[i]) ++i;              // kb < sum_end[kSumPairs - 1]
              ma = more + i;
              mb = more + kSumPairs + i;
              k0 = (i > 0 ? kb - p.sum_end[i - 1] : kb) * kElemsPerKB;
            }
            if (PAIR && second) {
              const int half = kb - num_kb1 >= num_kb2 ? 1 : 0, k2 = k0 - half * num_kb2 * kElemsPerKB;
              tma_load_cg<CG>(sa, half ? more : &tmA2, &full_bar[stage], k2, m0);
              tma_load_cg<CG>(sb, &tmB2, &full_bar[stage], k2, half == static_cast<int>(rank) ? n0 : p.N);
              if (++stage == C::kStages) { stage = 0; phase ^= 1; }
              continue;
            }
            if (BATCH) {
              tma_load3_cg<CG>(sa, ma, &full_bar[stage], k0, m0, bidx);
              tma_load3_cg<CG>(sb, mb, &full_bar[stage], k0, n0, bidx);
              if (++stage == C::kStages) { stage = 0; phase ^= 1; }
              continue;
            }
            if (A_MN) {          // stored [K rows][M cols]: two [64 k x 64 m] panels
              tma_load_cg<CG>(sa, ma, &full_bar[stage], m0, k0);
              tma_load_cg<CG>(sa + kPanelBytes, ma, &full_bar[stage], m0 + 64, k0);
            } else {
              tma_load_cg<CG>(sa, ma, &full_bar[stage], k0, m0);
            }
            if (B_MN) {
#pragma unroll
              for (int pn = 0; pn < C::kBPanels; ++pn)
                tma_load_cg<CG>(sb + pn * kPanelBytes, mb, &full_bar[stage], n0 + pn * 64, k0);
            } else {
              tma_load_cg<CG>(sb, mb, &full_bar[stage], k0, n0);
            }
            if (++stage == C::kStages) { stage = 0; phase ^= 1; }
          }
          if (!kRanges) break;
        }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer (leader CTA only) ================================
    if (leader && elect_one()) {
      constexpr uint32_t idesc = FP8 ? ((1u << 4) | ((static_cast<uint32_t>(BN) >> 3) << 17) | ((static_cast<uint32_t>(CG * BLOCK_M) >> 4) << 24))
                                     : make_idesc_tc(CG * BLOCK_M, BN, A_MN, B_MN);          // e4m3 x e4m3 (format code 0) -> fp32
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int w = unit; w < num_work; w += num_units) {
        TileCoord c{0, 0};
        const int n_end = range_of(w, c);
        for (; c.n_blk < n_end; ++c.n_blk) {
          mbar_wait(&tmem_empty[acc], acc_phase ^ 1);
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN;
          const int kb_lo = BATCH ? 0 : (w % splits) * kb_per_split, kb_hi = BATCH ? num_kb : min(num_kb, kb_lo + kb_per_split);
          for (int kb = kb_lo; kb < kb_hi; ++kb) {
            mbar_wait(&full_bar[stage], phase);
            tc_fence_after();
            const uint32_t a_addr = smem_u32(smem + stage * C::kStageBytes);
            const uint32_t b_addr = a_addr + kABytes;
#pragma unroll
            for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
              // K-major: 16 contraction elements = 32 bytes along the swizzled row; MN-major: 16 contraction rows = 2048 B
              const uint64_t adesc = A_MN ? make_smem_desc_sw128_mn(a_addr + k * UMMA_K * 128, kPanelBytes)
                                          : make_smem_desc_sw128(a_addr + k * UMMA_K * 2);
              const uint64_t bdesc = B_MN ? make_smem_desc_sw128_mn(b_addr + k * UMMA_K * 128, kPanelBytes)
                                          : make_smem_desc_sw128(b_addr + k * UMMA_K * 2);
              if (FP8) umma_fp8<CG>(d_tmem, adesc, bdesc, idesc, ((kb - kb_lo) | k) != 0 ? 1u : 0u);
              else umma_bf16<CG>(d_tmem, adesc, bdesc, idesc, ((kb - kb_lo) | k) != 0 ? 1u : 0u);
            }
            umma_commit_cg<CG>(&empty_bar[stage], pair);  // smem stage reusable once these MMAs retire
            if (++stage == C::kStages) { stage = 0; phase ^= 1; }
          }
          umma_commit_cg<CG>(&tmem_full[acc], pair);      // accumulator complete -> epilogue (of both CTAs)
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else {
    // ================================ epilogue (every CTA: its own 128 rows) ================================
    const int quad = warp & 3;                          // TMEM lane quadrant this warp may read
    const int row_in_tile = quad * 32 + lane;
    const int epi_tid = threadIdx.x - 64, group = (warp - 2) >> 2;      // the two warps of a quadrant take alternate chunks
    int acc = 0;
    uint32_t acc_phase = 0;
    uint8_t* slab = smem + C::kStagingOff + (warp - 2) * (EPI == EPI_DSWIGLU ? 2 : 1) * kSlabBytes;
    const bool bias_vec = CAT || (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
    // the accumulator has been read by this warp
    auto release_acc = [&]() {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_leader(&tmem_empty[acc]);
        else mbar_arrive(&tmem_empty[acc]);
      }
    };
    // 64 packed columns of this thread's row -> slab -> global
    auto store_slab_to = [&](const CUtensorMap* to, const uint32_t (&pk)[32], int col, int row0, int b) {
      if (lane == 0) tma_store_wait_read<0>();                          // the warp's previous store has drained
      __syncwarp();
      uint8_t* rowp = slab + lane * 128;
#pragma unroll
      for (int q8 = 0; q8 < 8; ++q8)
        *reinterpret_cast<uint4*>(rowp + ((q8 ^ (lane & 7)) * 16)) = make_uint4(pk[q8 * 4], pk[q8 * 4 + 1], pk[q8 * 4 + 2], pk[q8 * 4 + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (BATCH) tma_store_3d(to, slab, col, row0, b);
        else tma_store_2d(to, slab, col, row0);
        tma_store_commit();
      }
    };
    auto store_slab = [&](const uint32_t (&pk)[32], int col, int row0, int b) { store_slab_to(&tmD, pk, col, row0, b); };
    // EPI_DSWIGLU: gate and up of a chunk arrive in the warp's two slabs ahead of its sums and leave as their gradients
    uint64_t* in_bar = reinterpret_cast<uint64_t*>(smem + C::kBarOff + 256) + (warp - 2);
    uint32_t in_phase = 0;
    auto chunk_at = [&](int w, int it, int& col0, int& row0) {
      const TileCoord c = tile_coord(w, num_m, num_n);
      col0 = c.n_blk * BN + (it * 2 + group) * 64;
      row0 = (c.m_tile * CG + static_cast<int>(rank)) * BLOCK_M + quad * 32;
      return col0 < p.N && row0 < p.M;
    };
    auto fetch = [&](int w, int it) {
      int col0, row0;
      if (w < num_work && chunk_at(w, it, col0, row0) && lane == 0) {
        tma_store_wait_read<0>();                          // the slabs' last contents have left
        mbar_arrive_expect_tx(in_bar, 2 * kSlabBytes);
        tma_load_2d(slab, more, in_bar, col0, row0);
        tma_load_2d(slab + kSlabBytes, more + 1, in_bar, col0, row0);
      }
    };
    if (EPI == EPI_DSWIGLU) fetch(unit, 0);
    for (int w = unit; w < num_work; w += num_units) {
      const int tile_id = BATCH ? w % tiles_per_batch : w / splits;
      const int bidx = BATCH ? w / tiles_per_batch : 0;
      (void)bidx;
      TileCoord c = GROUPED || kRanges ? TileCoord{0, 0} : tile_coord(tile_id, num_m, num_n);
      const int n_end = range_of(w, c);
      const int which = CAT ? product_of(c.n_blk) : 0;
      const int n_cols = CAT ? cat->n[which] : p.N;
      const __nv_bfloat16* bias = CAT ? cat->bias[which] : p.bias;
      const int m_blk = c.m_tile * CG + static_cast<int>(rank);
      int row = m_blk * BLOCK_M + row_in_tile;
      int row_end = p.M;
      if (GROUPED) {
        const int mt = w / num_n;
        c.n_blk = w - mt * num_n;
        row = __ldg(p.grp_tiles + 3 * mt + 1) + row_in_tile;
        row_end = __ldg(p.grp_tiles + 3 * mt + 2);
      }
      const bool row_ok = row < row_end;
      if (EPI == EPI_LOGPROB) {
        // per row and warp group: largest logit, sum of exponentials, sum of exponential times logit and the target's logit over the item's columns
        constexpr float kLog2e = 1.4426950408889634f;
        const int target = row_ok ? p.targets[row] : -1;
        float run_max = -INFINITY, run_sum = 0.f, run_ez = 0.f, tgt = -INFINITY;
        for (; c.n_blk < n_end; ++c.n_blk) {
          mbar_wait(&tmem_full[acc], acc_phase);
          tc_fence_after();
          const uint32_t t_acc = tmem_base + acc * BN + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
          for (int it = 0; it < BN / 128; ++it) {
            uint32_t v[2][32];
            tmem_ld_32x32b_x32(t_acc + (it * 2 + group) * 64, v[0]);
            tmem_ld_32x32b_x32(t_acc + (it * 2 + group) * 64 + 32, v[1]);
            tmem_ld_wait();
            if (it == BN / 128 - 1) release_acc();
            const int col0 = c.n_blk * BN + (it * 2 + group) * 64;
            if (p.logits != nullptr && row_ok) {
              float* to = p.logits + static_cast<size_t>(row) * p.N + col0;
#pragma unroll
              for (int j = 0; j < 64; j += 8)
                if (col0 + j < p.N) stg_v8(to + j, &v[j >> 5][j & 31]);
            }
            float cmax = -INFINITY;
#pragma unroll
            for (int j = 0; j < 64; ++j) {
              float z = __uint_as_float(v[j >> 5][j & 31]) * p.alpha;
              z = col0 + j < p.N ? z : -INFINITY;
              v[j >> 5][j & 31] = __float_as_uint(z);
              cmax = fmaxf(cmax, z);
              if (col0 + j == target) tgt = z;
            }
            const float new_max = fmaxf(run_max, cmax);
            if (new_max > -INFINITY) {
              const float corr = exp2f((run_max - new_max) * kLog2e), mb = new_max * kLog2e;      // exp2(-inf) = 0 on the first chunk
              run_sum *= corr;
              run_ez *= corr;
#pragma unroll
              for (int j = 0; j < 64; ++j) {
                const float z = __uint_as_float(v[j >> 5][j & 31]), e = exp2f(fmaf(z, kLog2e, -mb));
                run_sum += e;
                run_ez = fmaf(e, z == -INFINITY ? 0.f : z, run_ez);
              }
              run_max = new_max;
            }
          }
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        if (row_ok)
          reinterpret_cast<float4*>(p.out_f32)[static_cast<size_t>((w / num_m) * 2 + group) * p.M + row] = make_float4(run_max, run_sum, run_ez, tgt);
        continue;
      }
      mbar_wait(&tmem_full[acc], acc_phase);
      tc_fence_after();
      const uint32_t t_acc = tmem_base + acc * BN + (static_cast<uint32_t>(quad * 32) << 16);
      uint32_t sw_packed[32];
      (void)sw_packed;
      float dl_lse = 0.f, dl_g = 0.f;
      int dl_target = -1;
      if (EPI == EPI_DLOGITS && row_ok) {
        dl_lse = p.lse[row];
        dl_g = p.grad[row] * p.alpha;                       // d logp / d logit carries the 1 / T factor
        dl_target = p.targets[row];
      }
      if (CLUSTER) {
        // ---- split-K by a cluster: the partial tile takes the place of the operands, all of which have been read, in the workspace's layout below ----
        float* mine = reinterpret_cast<float*>(smem) + row_in_tile * 4;
#pragma unroll 1
        for (int ch = group; ch < BN / 32; ch += 2) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_acc + ch * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(mine + (ch * 8 + (j >> 2)) * (BLOCK_M * 4)) =
                make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
        }
        break;                                             // one tile per block
      }
      if (SPLIT) {
        // ---- split-K: park the fp32 partial tile, the last CTA of the tile reduces all partials in split order ----
        const long tile_elems = static_cast<long>(BLOCK_M) * BN;
        // workspace tile layout [BN / 4 column groups][128 rows][4]: a warp's 32 rows of one column group are 512 contiguous
        // bytes, for the partial stores here and for the reduction's loads below
        const int part_id = tile_id * CG + static_cast<int>(rank), num_parts = num_m * num_n * CG;      // a block's half of a pair's tile
        float* mine = p.ws + (static_cast<long>(w % splits) * num_parts + part_id) * tile_elems + row_in_tile * 4;
#pragma unroll 1
        for (int ch = group; ch < BN / 32; ch += 2) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_acc + ch * 32, v);
          tmem_ld_wait();
          if (ch + 2 >= BN / 32) release_acc();
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            __stcg(reinterpret_cast<float4*>(mine + (ch * 8 + (j >> 2)) * (BLOCK_M * 4)),
                   make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])));
        }
        __threadfence();                                   // this thread's partial is visible device-wide ...
        named_barrier_sync(1, kEpiThreads);                // ... and so is every other epilogue thread's
        if (epi_tid == 0) {
          const int old = atomicAdd(p.counters + part_id, 1);
          const int last = (old == splits - 1) ? 1 : 0;
          if (last) p.counters[part_id] = 0;               // self-reset for the next launch
          __threadfence();
          *s_last = last;
        }
        named_barrier_sync(2, kEpiThreads);
        if (*s_last && row_ok) {
          const float* base = p.ws + static_cast<long>(part_id) * tile_elems + row_in_tile * 4;
          const long split_stride = static_cast<long>(num_parts) * tile_elems;
          __nv_bfloat16* orow = p.out_bf16 + static_cast<long>(row) * p.out_stride + c.n_blk * BN;
#pragma unroll 1
          for (int c0 = group * 32; c0 < BN; c0 += 64) {
            if (c.n_blk * BN + c0 >= p.N) break;
            float acc[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) acc[e] = 0.f;
#pragma unroll 1
            for (int sp = 0; sp < splits; ++sp) {            // fixed order -> deterministic; 8 independent 16-byte loads in flight
              const float* b = base + sp * split_stride + (c0 >> 2) * (BLOCK_M * 4);
              float4 x[8];
#pragma unroll
              for (int q = 0; q < 8; ++q) x[q] = __ldcg(reinterpret_cast<const float4*>(b + q * (BLOCK_M * 4)));
#pragma unroll
              for (int q = 0; q < 8; ++q) { acc[4 * q] += x[q].x; acc[4 * q + 1] += x[q].y; acc[4 * q + 2] += x[q].z; acc[4 * q + 3] += x[q].w; }
            }
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              if (c.n_blk * BN + c0 + j < p.N) {             // N % 8 == 0
                float s8[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) s8[e] = acc[j + e] * p.alpha;
                if (p.bias != nullptr) {
                  const uint4 bv = *reinterpret_cast<const uint4*>(p.bias + c.n_blk * BN + c0 + j);      // bias 16-byte aligned
                  const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const float2 bf = unpack_bf16x2(bw[e]);
                    s8[2 * e] += bf.x;
                    s8[2 * e + 1] += bf.y;
                  }
                }
                *reinterpret_cast<uint4*>(orow + c0 + j) = make_uint4(pack_bf16x2(s8[0], s8[1]), pack_bf16x2(s8[2], s8[3]),
                                                                      pack_bf16x2(s8[4], s8[5]), pack_bf16x2(s8[6], s8[7]));
              }
            }
          }
        }
        named_barrier_sync(1, kEpiThreads);                // s_last is rewritten by the next work item
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        continue;
      }
      if (EPI == EPI_DSWIGLU) {
        // the gradient of the activation is rounded as its own GEMM would leave it, then d gate = g * up * (s + gate s (1 - s)), d up = g * gate * s
#pragma unroll 1
        for (int it = 0; it < BN / 128; ++it) {
          int col0, row0;
          const bool ok = chunk_at(w, it, col0, row0);
          uint32_t v[2][32];
          tmem_ld_32x32b_x32(t_acc + (it * 2 + group) * 64, v[0]);
          tmem_ld_32x32b_x32(t_acc + (it * 2 + group) * 64 + 32, v[1]);
          tmem_ld_wait();
          if (it == BN / 128 - 1) release_acc();
          if (ok) {
            mbar_wait(in_bar, in_phase);
            in_phase ^= 1;
            uint8_t* rg = slab + lane * 128;
#pragma unroll
            for (int q8 = 0; q8 < 8; ++q8) {
              uint4* pg = reinterpret_cast<uint4*>(rg + ((q8 ^ (lane & 7)) * 16));
              uint4* pu = reinterpret_cast<uint4*>(rg + kSlabBytes + ((q8 ^ (lane & 7)) * 16));
              const uint4 g4 = *pg, u4 = *pu;
              const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w}, uw[4] = {u4.x, u4.y, u4.z, u4.w};
              uint32_t dg[4], du[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int j = q8 * 8 + 2 * e;
                const float2 o = unpack_bf16x2(pack_bf16x2(__uint_as_float(v[j >> 5][j & 31]), __uint_as_float(v[j >> 5][(j & 31) + 1])));
                const float2 a = unpack_bf16x2(gw[e]), b = unpack_bf16x2(uw[e]);
                const float s0 = 1.f / (1.f + __expf(-a.x)), s1 = 1.f / (1.f + __expf(-a.y));
                dg[e] = pack_bf16x2(o.x * b.x * (s0 + a.x * s0 * (1.f - s0)), o.y * b.y * (s1 + a.y * s1 * (1.f - s1)));
                du[e] = pack_bf16x2(o.x * a.x * s0, o.y * a.y * s1);
              }
              *pg = make_uint4(dg[0], dg[1], dg[2], dg[3]);
              *pu = make_uint4(du[0], du[1], du[2], du[3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmD, slab, col0, row0);
              tma_store_2d(more + 2, slab + kSlabBytes, col0, row0);
              tma_store_commit();
            }
          }
          if (it + 1 < BN / 128) fetch(w, it + 1);
          else fetch(w + num_units, 0);
        }
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        continue;
      }
      if (PAIR) {                                           // group 0 takes features 0 .. 63 of the tile, group 1 the others
        constexpr int kKeep = EPI == EPI_SWIGLU_KEEP ? 32 : 1;
        uint32_t pk[32], gk[kKeep], uk[kKeep];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t g[32], u[32];
          tmem_ld_32x32b_x32(t_acc + group * 64 + h * 32, g);
          tmem_ld_32x32b_x32(t_acc + BN / 2 + group * 64 + h * 32, u);
          tmem_ld_wait();
          if (h == 1) release_acc();
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            // gate and up are rounded as the two projections' own GEMMs leave them and combined as swiglu_kernel combines them: log-probabilities
            // taken outside autograd round as the training forward does, the ratio of an unchanged policy stays 1
            const uint32_t g2 = pack_bf16x2(__uint_as_float(g[j]), __uint_as_float(g[j + 1])), u2 = pack_bf16x2(__uint_as_float(u[j]), __uint_as_float(u[j + 1]));
            const float2 gr = unpack_bf16x2(g2), ur = unpack_bf16x2(u2);
            if (EPI == EPI_SWIGLU_KEEP) {
              gk[(h * 16 + j / 2) % kKeep] = g2;
              uk[(h * 16 + j / 2) % kKeep] = u2;
            }
            pk[h * 16 + j / 2] = pack_bf16x2(gr.x / (1.f + __expf(-gr.x)) * ur.x, gr.y / (1.f + __expf(-gr.y)) * ur.y);
          }
        }
        const int col = c.n_blk * (BN / 2) + group * 64;
        if (col < p.N / 2 && m_blk * BLOCK_M + quad * 32 < p.M) {
          store_slab(pk, col, m_blk * BLOCK_M + quad * 32, 0);
          if constexpr (EPI == EPI_SWIGLU_KEEP) {
            store_slab_to(more + 1, gk, col, m_blk * BLOCK_M + quad * 32, 0);
            store_slab_to(more + 2, uk, col, m_blk * BLOCK_M + quad * 32, 0);
          }
        }
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        continue;
      }
#pragma unroll 1
      for (int it = 0;; ++it) {
        // SwiGLU: two neighbouring chunks make one output slab and stay with one warp
        const int ch = EPI == EPI_SWIGLU ? (it >> 1) * 4 + group * 2 + (it & 1) : it * 2 + group;
        if (ch >= BN / 64) {
          if (it == 0) release_acc();                   // no chunk for this warp
          break;
        }
        uint32_t v[2][32];
        float gate_scale = 0.f, up_scale = 0.f;          // FP8 SwiGLU: lane l holds those of the chunk's columns l and 32 + l
        if (FP8 && EPI == EPI_SWIGLU) {
          const int cl = c.n_blk * BN + ch * 64 + lane;
          if (cl < p.N) gate_scale = __ldg(p.col_scale + cl);
          if (cl + 32 < p.N) up_scale = __ldg(p.col_scale + cl + 32);
        }
        // A residual is read a row per thread as whole sectors, ahead of the sums: 128 bytes in 0.4 us that a tile's epilogue
        // has to spare.  A form of its own: behind a run-time branch of the plain one it cost other GEMMs 2 %.
        constexpr bool kResidual = EPI == EPI_RESIDUAL;
        uint4 rs[8];
        if (kResidual && row_ok) {
          const int cl = c.n_blk * BN + ch * 64;
          const uint4* from = reinterpret_cast<const uint4*>(p.residual + static_cast<long>(row) * p.residual_stride + cl);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (cl + q * 8 < p.N) rs[q] = __ldg(from + q);
        }
        tmem_ld_32x32b_x32(t_acc + ch * 64, v[0]);
        tmem_ld_32x32b_x32(t_acc + ch * 64 + 32, v[1]);
        tmem_ld_wait();
        if ((EPI == EPI_SWIGLU ? ((it + 1) >> 1) * 4 + group * 2 + ((it + 1) & 1) : ch + 2) >= BN / 64) release_acc();      // its last one
        const int col0 = c.n_blk * BN + ch * 64;
        if (EPI == EPI_GRP_RELU2) {
          // grouped up projection with the squared ReLU formed here: a chunk yields 64 activations of this row
          const float rw = p.row_scale != nullptr && row_ok ? p.row_scale[row] : 1.f;
          uint32_t pk[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float a0 = fmaxf(rw * __uint_as_float(v[j >> 4][(j & 15) * 2]), 0.f), a1 = fmaxf(rw * __uint_as_float(v[j >> 4][(j & 15) * 2 + 1]), 0.f);
            pk[j] = pack_bf16x2(a0 * a0, a1 * a1);
          }
          warp_rows_out(slab, pk, lane, [&](int, int r, int q, const uint4& x) {      // N % 8 == 0
            const int rr = row - lane + r, col = col0 + q * 8;
            if (rr < row_end && col < p.N) *reinterpret_cast<uint4*>(p.out_bf16 + static_cast<long>(rr) * p.out_stride + col) = x;
          });
        } else if (EPI == EPI_GRP_SWIGLU) {
          // grouped gate / up projection with the SwiGLU formed here: B rows are interleaved per 32 features ([32 gate | 32 up]
          // in every 64-column chunk), so a chunk yields 32 activations of this row: 64 contiguous bytes
          const int f0 = c.n_blk * (BN / 2) + ch * 32;
          if (f0 < p.N / 2) {
            const float rw = p.row_scale != nullptr && row_ok ? p.row_scale[row] : 1.f;      // a weight on the expert's input: gate and up scale with it
            uint32_t pk[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float g0 = rw * __uint_as_float(v[0][2 * e]), g1 = rw * __uint_as_float(v[0][2 * e + 1]);
              const float u0 = rw * __uint_as_float(v[1][2 * e]), u1 = rw * __uint_as_float(v[1][2 * e + 1]);
              pk[e] = pack_bf16x2(g0 / (1.f + __expf(-g0)) * u0, g1 / (1.f + __expf(-g1)) * u1);
            }
            warp_rows_out(slab, pk, lane, [&](int, int r, int q, const uint4& x) {
              const int rr = row - lane + r;
              if (rr < row_end) *reinterpret_cast<uint4*>(p.out_bf16 + static_cast<long>(rr) * p.out_stride + f0 + q * 8) = x;
            });
          }
        } else if (EPI == EPI_F32) {
          // fp32 row-major out (+)= alpha * acc: 128 contiguous bytes of four rows at a time; N % 4 == 0 (checked on the host)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int cl = col0 + h * 32 + (lane & 7) * 4, r0 = row - lane + (lane >> 3);      // this lane's column and first row
            float4* dst = reinterpret_cast<float4*>(p.out_f32 + static_cast<long>(r0) * p.out_f32_stride + cl);
            float4 old[8];
            if (!GROUPED && p.accumulate) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (r0 + 4 * i < row_end && cl < p.N) old[i] = dst[i * p.out_f32_stride];
            }
            uint32_t x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = __float_as_uint(__uint_as_float(v[h][j]) * p.alpha);
            warp_rows_out(slab, x, lane, [&](int i, int, int, const uint4& y) {
              if (r0 + 4 * i >= row_end || cl >= p.N) return;
              float4 o = make_float4(__uint_as_float(y.x), __uint_as_float(y.y), __uint_as_float(y.z), __uint_as_float(y.w));
              if (!GROUPED && p.accumulate) {
                o.x += old[i].x; o.y += old[i].y; o.z += old[i].z; o.w += old[i].w;
              }
              dst[i * p.out_f32_stride] = o;
            });
          }
        } else if (EPI == EPI_SWIGLU) {
          // every 64-column chunk of the accumulator is [32 gate | 32 up] of the same 32 features (weight rows interleaved at
          // weight-refresh time, parallel/weight_sync.py): silu(g) * u is formed in registers, two chunks make one 64-wide
          // output slab -- the [tokens, 2F] gate_up tensor never exists
          constexpr float kLog2e = 1.4426950408889634f;
          const float rs8 = (FP8 && row_ok) ? p.row_scale[row] : 1.f;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            float g0 = __uint_as_float(v[0][j]), g1 = __uint_as_float(v[0][j + 1]);
            float u0 = __uint_as_float(v[1][j]), u1 = __uint_as_float(v[1][j + 1]);
            if (FP8) {
              g0 *= rs8 * __shfl_sync(0xffffffffu, gate_scale, j); g1 *= rs8 * __shfl_sync(0xffffffffu, gate_scale, j + 1);
              u0 *= rs8 * __shfl_sync(0xffffffffu, up_scale, j); u1 *= rs8 * __shfl_sync(0xffffffffu, up_scale, j + 1);
            }
            const uint32_t pk = pack_bf16x2(g0 / (1.f + exp2f(-g0 * kLog2e)) * u0, g1 / (1.f + exp2f(-g1 * kLog2e)) * u1);
            if ((ch & 1) == 0) sw_packed[j / 2] = pk;     // static indices: the array stays in registers
            else sw_packed[16 + j / 2] = pk;
          }
          if ((ch & 1) && c.n_blk * (BN / 2) + (ch >> 1) * 64 < p.N / 2 && m_blk * BLOCK_M + quad * 32 < p.M)
            store_slab(sw_packed, c.n_blk * (BN / 2) + (ch >> 1) * 64, m_blk * BLOCK_M + quad * 32, 0);
        } else {
          uint32_t packed[32];
#pragma unroll
          for (int j = 0; j < 64; j += 8) {
            const int col = col0 + j;
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[j >> 5][(j & 31) + e]) * p.alpha;
            if (FP8) {
              const float rs = row_ok ? p.row_scale[row] : 0.f;
#pragma unroll
              for (int e = 0; e < 8; ++e) x[e] *= rs * ((col + e < p.N) ? p.col_scale[col + e] : 0.f);
            }
            if (EPI == EPI_DLOGITS) {
#pragma unroll
              for (int e = 0; e < 8; ++e) x[e] = ((col + e == dl_target ? 1.f : 0.f) - exp2f((x[e] - dl_lse) * 1.4426950408889634f)) * dl_g;
            }
            if (EPI != EPI_DLOGITS && bias != nullptr && col < n_cols) {        // N % 8 == 0
              uint32_t bw[4];
              if (bias_vec) {
                const uint4 bv = __ldg(reinterpret_cast<const uint4*>(bias + col));
                bw[0] = bv.x; bw[1] = bv.y; bw[2] = bv.z; bw[3] = bv.w;
              } else {
                const uint16_t* b16 = reinterpret_cast<const uint16_t*>(bias + col);
#pragma unroll
                for (int e = 0; e < 4; ++e) bw[e] = b16[2 * e] | (static_cast<uint32_t>(b16[2 * e + 1]) << 16);
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 bf = unpack_bf16x2(bw[e]);
                x[2 * e] += bf.x;
                x[2 * e + 1] += bf.y;
              }
            }
            if (EPI != EPI_DLOGITS && p.act == 1) {
#pragma unroll
              for (int e = 0; e < 8; ++e) x[e] = gelu_erf_tc(x[e]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) packed[j / 2 + e] = pack_bf16x2(x[2 * e], x[2 * e + 1]);
            if (kResidual) {       // rounded, then added and rounded, as by a kernel of its own
              const uint32_t r[4] = {rs[j / 8].x, rs[j / 8].y, rs[j / 8].z, rs[j / 8].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 y = unpack_bf16x2(packed[j / 2 + e]), z = unpack_bf16x2(r[e]);
                packed[j / 2 + e] = pack_bf16x2(y.x + z.x, y.y + z.y);
              }
            }
          }
          if (col0 < n_cols && m_blk * BLOCK_M + quad * 32 < p.M) store_slab_to(CAT ? more + 3 * kCatMax + which : &tmD, packed, col0, m_blk * BLOCK_M + quad * 32, bidx);
        }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (!kPlainStores && !SPLIT && lane == 0) tma_store_wait<0>();
  }

  if (CLUSTER) {
    // every block sums a share of the tile over the cluster's parts, in split order
    __syncwarp();
    cluster_sync_all();
    const TileCoord c = tile_coord(unit / splits, num_m, num_n);
    const int me = unit % splits, units = BLOCK_M * BN / 8;                  // a unit: eight columns of a row
    const uint32_t part = smem_u32(smem);
    for (int u = units * me / splits + threadIdx.x; u < units * (me + 1) / splits; u += kThreads) {
      const int row = (c.m_tile * CG + static_cast<int>(rank)) * BLOCK_M + (u & (BLOCK_M - 1)), g8 = u / BLOCK_M, col = c.n_blk * BN + g8 * 8;
      if (row >= p.M || col >= p.N) continue;              // N % 8 == 0
      const uint32_t at = part + (g8 * 2 * BLOCK_M + (u & (BLOCK_M - 1))) * 16;
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll 1
      for (int s0 = 0; s0 < splits; s0 += 4) {
        float4 x[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (s0 + i < splits) {
            x[i][0] = ld_cluster_f4(at, (s0 + i) * CG + rank);
            x[i][1] = ld_cluster_f4(at + BLOCK_M * 16, (s0 + i) * CG + rank);
          }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (s0 + i < splits) {
            acc[0] += x[i][0].x; acc[1] += x[i][0].y; acc[2] += x[i][0].z; acc[3] += x[i][0].w;
            acc[4] += x[i][1].x; acc[5] += x[i][1].y; acc[6] += x[i][1].z; acc[7] += x[i][1].w;
          }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] *= p.alpha;
      if (p.bias != nullptr) {
        const uint4 bv = *reinterpret_cast<const uint4*>(p.bias + col);      // bias 16-byte aligned
        const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 bf = unpack_bf16x2(bw[e]);
          acc[2 * e] += bf.x;
          acc[2 * e + 1] += bf.y;
        }
      }
      if (MULTI && p.transposed) {                         // neighbouring threads hold neighbouring rows
#pragma unroll
        for (int e = 0; e < 8; ++e) p.out_bf16[static_cast<long>(col + e) * p.out_stride + row] = __float2bfloat16(acc[e]);
        continue;
      }
      *reinterpret_cast<uint4*>(p.out_bf16 + static_cast<long>(row) * p.out_stride + col) =
          make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]), pack_bf16x2(acc[6], acc[7]));
    }
    __syncwarp();
  }
  tc_fence_before();
  if (CLUSTER) cluster_sync_all();          // nobody leaves while others read its part
  else if (CG == 2) cluster_sync_all();     // nobody leaves (or frees TMEM) while the peer can still signal / read it
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_cg<CG>(tmem_base, C::kTmemCols);
  }
}

template <int BN, bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_cg1_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2,
                   const __grid_constant__ CUtensorMap tmD, const TcParams p) {
  gemm_tc_body<1, BN, A_MN, B_MN, EPI>(tmA, tmB, tmA2, tmB2, tmD, p);
}
template <int BN, bool A_MN, bool B_MN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_cg2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2,
                   const __grid_constant__ CUtensorMap tmD, const TcParams p) {
  gemm_tc_body<2, BN, A_MN, B_MN, EPI>(tmA, tmB, tmA2, tmB2, tmD, p);
}

template <int N>
struct TcMaps { CUtensorMap m[N]; };      // as many as a kernel reads: they are launch parameters too

// EPI: EPI_SWIGLU, or EPI_SWIGLU_KEEP where gate and up are wanted too (training); more = {the up adapter's columns, gate, up}.  Two GEMMs and an activation
// pass move 2.4 times as much memory, the pass alone 54 us of traffic at 6601 x 8960; three stores a tile hide behind its 26 blocks of contraction.
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBg, const __grid_constant__ CUtensorMap tmBu,
                    const __grid_constant__ CUtensorMap tmA2g, const __grid_constant__ CUtensorMap tmB2g, const __grid_constant__ CUtensorMap tmB2u,
                    const __grid_constant__ CUtensorMap tmD, const __grid_constant__ TcMaps<EPI == EPI_SWIGLU_KEEP ? 3 : 1> more, const TcParams p) {
  const bool up = cluster_ctarank() != 0;
  gemm_tc_body<2, 256, false, false, EPI, false, false, false, false, true>(tmA, up ? tmBu : tmBg, tmA2g, up ? tmB2u : tmB2g, tmD, p, more.m);
}

// (d gate, d up) of the SwiGLU from d y of the projection behind it: d act = dY W + T A, which never is in memory; more = {gate, up, d up}.
// Gate and up of a chunk (32 rows x 64 columns of each, a warp's own) are fetched while its sums are formed and overwritten by their gradients, so that the
// epilogue holds two slabs a warp and waits for nothing of another warp; one stage of the ring less pays for the second slab.
// With this, the kept gate and up and sums in one accumulator a decoder layer's forward and backward over 6601 tokens takes 1724 us, 1862 before.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_dswiglu_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA2,
                       const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmD, const __grid_constant__ TcMaps<3> more,
                       const TcParams p) {
  gemm_tc_body<2, 256, false, true, EPI_DSWIGLU>(tmA, tmB, tmA2, tmB2, tmD, p, more.m);
}

// D = the sum of up to kSumPairs products A_i [M, K_i] B_i [K_i, N] in one accumulator: the gradient of an input that several projections share, without a
// result, an addition and a rounding per projection (6601 x 1536: 60 MB each time)
template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_sum_kernel(const __grid_constant__ TcMaps<2 * kSumPairs> maps, const __grid_constant__ CUtensorMap tmD, const TcParams p) {
  gemm_tc_body<2, BN, false, true, EPI_BF16, false, false, false, false, false, false, true>(tmD, tmD, tmD, tmD, tmD, p, maps.m);
}
template <int BN>
static cudaError_t launch_sum(const TcMaps<2 * kSumPairs>& maps, const CUtensorMap& tmD, const TcParams& p, int num_sms, cudaStream_t stream) {
  using C = Cfg<2, BN, true>;
  auto kern = gemm_tc_sum_kernel<BN>;
  static nrl::PerDevice<bool> configured;
  if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
  int units = ((p.M + 255) / 256) * ((p.N + BN - 1) / BN);
  if (units > num_sms / 2) units = num_sms / 2;
  if (units < 1) units = 1;
  launch_dependent(kern, 2 * units, kThreads, C::kTotal, stream, maps, tmD, p);
  return cudaGetLastError();
}

// D_i = A B_i^T + A2_i B2_i^T (+ bias_i): the projections of one input (query, key, value) in one launch, whose column tiles lie side by side: one start and one
// last wave for all.  us, a launch each -> one (rows 250, 800, 3300, 6601, 24 571, 32 768): 3 x 1024 features of 1024: 23 -> 7.4, 24 -> 10, 39 -> 21, 47 -> 31, 127 -> 106, 156 -> 138;
// 1536 + 256 + 256 of 1536 with adapters of rank 64: 31 -> 10, 30 -> 10, 39 -> 20, 47 -> 30, 131 -> 108, 164 -> 141; 3584 + 512 + 512 of 3584: 65 -> 17, 54 -> 24, 92 -> 81,
// 165 -> 146, 626 -> 608, 788 -> 759.
template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_cat_cg1_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ TcMaps<4 * kCatMax> maps, const TcParams p, const __grid_constant__ TcCat cat) {
  gemm_tc_body<1, BN, false, false, EPI_BF16, false, false, false, false, false, false, false, true>(tmA, tmA, tmA, tmA, tmA, p, maps.m, 0, &cat);
}
template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_cat_cg2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ TcMaps<4 * kCatMax> maps, const TcParams p, const __grid_constant__ TcCat cat) {
  gemm_tc_body<2, BN, false, false, EPI_BF16, false, false, false, false, false, false, false, true>(tmA, tmA, tmA, tmA, tmA, p, maps.m, 0, &cat);
}
template <int CG, int BN>
static cudaError_t launch_cat(const CUtensorMap& tmA, const TcMaps<4 * kCatMax>& maps, const TcParams& p, const TcCat& cat, int num_sms, cudaStream_t stream) {
  using C = Cfg<CG, BN>;
  auto kern = CG == 2 ? gemm_tc_cat_cg2_kernel<BN> : gemm_tc_cat_cg1_kernel<BN>;
  static nrl::PerDevice<bool> configured;
  if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
  int units = (p.M + CG * BLOCK_M - 1) / (CG * BLOCK_M) * cat.end[kCatMax - 1];
  if (units > num_sms / CG) units = num_sms / CG;
  if (units < 1) units = 1;
  launch_dependent(kern, CG * units, kThreads, C::kTotal, stream, tmA, maps, p, cat);
  return cudaGetLastError();
}

// FORM: one kernel for each epilogue; with all three behind run-time branches in one kernel steps of 64 to 256 tokens took half a microsecond longer per GEMM
template <int BN, int FORM>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_grouped_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcParams p) {
  gemm_tc_body<1, BN, false, false, FORM, false, false, false, true>(tmA, tmB, tmA, tmB, tmA, p);
}
template <int BN, int FORM>
static cudaError_t launch_grouped_form(const CUtensorMap* maps, const TcParams& p, int units, cudaStream_t stream) {
  using C = Cfg<1, BN, false>;
  auto kern = gemm_tc_grouped_kernel<BN, FORM>;
  static nrl::PerDevice<bool> configured;
  if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
  launch_dependent(kern, units, kThreads, C::kTotal, stream, maps[0], maps[1], p);
  return cudaGetLastError();
}
template <int BN>
static cudaError_t launch_grouped(const CUtensorMap* maps, const TcParams& p, int max_tiles, int num_sms, cudaStream_t stream) {
  const int num_n = (p.N + BN - 1) / BN;
  long units = static_cast<long>(max_tiles) * num_n;
  if (units > num_sms) units = num_sms;
  if (units < 1) units = 1;
  const int n = static_cast<int>(units);
  if (p.out_bf16 == nullptr) return launch_grouped_form<BN, EPI_F32>(maps, p, n, stream);
  return p.act == 2 ? launch_grouped_form<BN, EPI_GRP_RELU2>(maps, p, n, stream) : launch_grouped_form<BN, EPI_GRP_SWIGLU>(maps, p, n, stream);
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_batched_cg1_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                           const __grid_constant__ CUtensorMap tmD, const TcParams p) {
  gemm_tc_body<1, BN, false, false, EPI_BF16, false, true>(tmA, tmB, tmA, tmB, tmD, p);
}
template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_batched_cg2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                           const __grid_constant__ CUtensorMap tmD, const TcParams p) {
  gemm_tc_body<2, BN, false, false, EPI_BF16, false, true>(tmA, tmB, tmA, tmB, tmD, p);
}
template <int BN, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_fp8_cg1_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const __grid_constant__ CUtensorMap tmD, const TcParams p) {
  gemm_tc_body<1, BN, false, false, EPI, false, false, true>(tmA, tmB, tmA, tmB, tmD, p);
}
template <int BN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_fp8_cg2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const __grid_constant__ CUtensorMap tmD, const TcParams p) {
  gemm_tc_body<2, BN, false, false, EPI, false, false, true>(tmA, tmB, tmA, tmB, tmD, p);
}
template <int CG, int BN, int EPI>
static cudaError_t launch_fp8(const CUtensorMap* maps, const TcParams& p, int num_sms, cudaStream_t stream) {
  using C = Cfg<CG, BN, false>;
  const int num_m = (p.M + CG * BLOCK_M - 1) / (CG * BLOCK_M), num_n = (p.N + BN - 1) / BN;
  int units = num_m * num_n;
  if (units > num_sms / CG) units = num_sms / CG;
  if (units < 1) units = 1;
  static nrl::PerDevice<bool> configured;
  if (CG == 1) {
    auto kern = gemm_tc_fp8_cg1_kernel<BN, EPI>;
    if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
    launch_dependent(kern, units, kThreads, C::kTotal, stream, maps[0], maps[1], maps[2], p);
  } else {
    auto kern = gemm_tc_fp8_cg2_kernel<BN, EPI>;
    if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
    launch_dependent(kern, 2 * units, kThreads, C::kTotal, stream, maps[0], maps[1], maps[2], p);
  }
  return cudaGetLastError();
}

template <int CG, int BN>
static cudaError_t launch_batched(const CUtensorMap* maps, const TcParams& p, int num_sms, cudaStream_t stream) {
  using C = Cfg<CG, BN, false>;
  const int num_m = (p.M + CG * BLOCK_M - 1) / (CG * BLOCK_M), num_n = (p.N + BN - 1) / BN;
  long units = static_cast<long>(num_m) * num_n * p.batch;
  if (units > num_sms / CG) units = num_sms / CG;
  if (units < 1) units = 1;
  static nrl::PerDevice<bool> configured;
  if (CG == 1) {
    auto kern = gemm_tc_batched_cg1_kernel<BN>;
    if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
    launch_dependent(kern, static_cast<int>(units), kThreads, C::kTotal, stream, maps[0], maps[1], maps[2], p);
  } else {
    auto kern = gemm_tc_batched_cg2_kernel<BN>;
    if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
    launch_dependent(kern, static_cast<int>(2 * units), kThreads, C::kTotal, stream, maps[0], maps[1], maps[2], p);
  }
  return cudaGetLastError();
}

template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_splitk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcParams p) {
  gemm_tc_body<1, BN, A_MN, B_MN, EPI_BF16, true>(tmA, tmB, tmA, tmB, tmA, p);
}

// The same with a tile's ranges in one cluster, which sums its parts through distributed shared memory: the workspace form passes them through L2, and its
// last block sums them alone while the others have left.  As many clusters as the GPU holds at a time; larger products and pairs of long ranges keep that form.
template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_splitk_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcParams p) {
  gemm_tc_body<1, BN, A_MN, B_MN, EPI_BF16, true, false, false, false, false, true>(tmA, tmB, tmA, tmB, tmA, p);
}

struct ClusterCounts { int plus_one[kMaxClusterSplits + 1]; };               // 0: not asked yet
// clusters of `blocks` blocks of a kernel that the current device runs at a time; the kernel may then use its shared memory there
template <class Kernel>
static int clusters_of(nrl::PerDevice<ClusterCounts>& counts, Kernel kernel, int smem, int blocks) {
  int& n = counts.here().plus_one[blocks];
  if (n == 0) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    n = 1 + (e == cudaSuccess ? clusters_at_a_time(kernel, kThreads, smem, blocks) : 0);
  }
  return n - 1;
}

// Several products with results at most a few tiles wide (the adapters' factors and inputs) in one launch: each of them alone leaves SMs idle and starts and
// ends for 5 us, as long as it works.  The products' tiles lie one after the other over the grid, every tile cut into the same number of ranges.
struct TcMulti {
  CUtensorMap a[kMultiMax], b[kMultiMax];
  int tiles[kMultiMax];                                    // up to and with the i-th product
  int M[kMultiMax], N[kMultiMax], K[kMultiMax];
  float alpha[kMultiMax];
  __nv_bfloat16* out[kMultiMax];
  long stride[kMultiMax];
  int transposed[kMultiMax];
};
template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_multi_kernel(const __grid_constant__ TcMulti m, const int splits) {
  int i = 0;
  while (static_cast<int>(blockIdx.x) >= m.tiles[i] * splits) ++i;      // the grid ends with the last product
  TcParams p{};
  p.M = m.M[i]; p.N = m.N[i]; p.K = m.K[i];
  p.alpha = m.alpha[i];
  p.splits = splits;
  p.out_bf16 = m.out[i];
  p.out_stride = m.stride[i];
  p.transposed = m.transposed[i];
  gemm_tc_body<1, 64, A_MN, B_MN, EPI_BF16, true, false, false, false, false, true, false, false, true>(m.a[i], m.b[i], m.a[i], m.b[i], m.a[i], p, nullptr,
                                                                                   i > 0 ? m.tiles[i - 1] * splits : 0);
}
template <bool A_MN, bool B_MN>
static int multi_clusters(int splits) {
  if (splits < 1 || splits > kMaxClusterSplits) return 0;
  static nrl::PerDevice<ClusterCounts> counts;
  return clusters_of(counts, gemm_tc_multi_kernel<A_MN, B_MN>, Cfg<1, 64, B_MN>::kTotal, splits);
}
template <bool A_MN, bool B_MN>
static cudaError_t launch_multi(const TcMulti& m, int n, int splits, cudaStream_t stream) {
  if (multi_clusters<A_MN, B_MN>(splits) < 1) return cudaErrorInvalidConfiguration;
  launch_dependent_clusters(gemm_tc_multi_kernel<A_MN, B_MN>, m.tiles[n - 1] * splits, kThreads, Cfg<1, 64, B_MN>::kTotal, stream, splits, m, splits);
  return cudaGetLastError();
}

// The same with pairs of blocks on a tile of 256 rows: a cluster is `splits` pairs, and each block sums rows of its own half.
template <int BN, bool B_MN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_split_pairs_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcParams p) {
  static_assert(Cfg<2, BN, B_MN>::kStagingOff >= BLOCK_M * BN * 4, "a part takes the place of the operands");
  gemm_tc_body<2, BN, false, B_MN, EPI_BF16, true, false, false, false, false, true>(tmA, tmB, tmA, tmB, tmA, p);
}
static_assert(Cfg<2, 128, true>::kTotal > kSmemBudget / 2 && Cfg<2, 128, false>::kTotal > kSmemBudget / 2 && Cfg<2, 192, true>::kTotal > kSmemBudget / 2 &&
              Cfg<2, 192, false>::kTotal > kSmemBudget / 2 && Cfg<2, 256, true>::kTotal > kSmemBudget / 2 && Cfg<2, 256, false>::kTotal > kSmemBudget / 2,
              "one block per SM in either form of B: nrl_gemm_tc_pair_clusters asks for one");
template <int BN, bool B_MN>
static int split_pairs_clusters(int splits) {
  if (splits < 2 || 2 * splits > kMaxClusterSplits) return 0;
  static nrl::PerDevice<ClusterCounts> counts;
  return clusters_of(counts, gemm_tc_split_pairs_kernel<BN, B_MN>, Cfg<2, BN, B_MN>::kTotal, 2 * splits);
}
// ... or passed through the workspace
template <int BN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_split_pairs_ws_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcParams p) {
  gemm_tc_body<2, BN, false, B_MN, EPI_BF16, true>(tmA, tmB, tmA, tmB, tmA, p);
}
template <int BN, bool B_MN>
static cudaError_t launch_split_pairs(const CUtensorMap* maps, const TcParams& p, bool clusters, int num_sms, cudaStream_t stream) {
  using C = Cfg<2, BN, B_MN>;
  const int tiles = ((p.M + 255) / 256) * ((p.N + BN - 1) / BN);
  if (clusters) {
    if (tiles > split_pairs_clusters<BN, B_MN>(p.splits)) return cudaErrorInvalidConfiguration;
    launch_dependent_clusters(gemm_tc_split_pairs_kernel<BN, B_MN>, tiles * p.splits * 2, kThreads, C::kTotal, stream, 2 * p.splits, maps[0], maps[1], p);
    return cudaGetLastError();
  }
  if (p.ws == nullptr || p.counters == nullptr) return cudaErrorInvalidValue;
  auto kern = gemm_tc_split_pairs_ws_kernel<BN, B_MN>;
  static nrl::PerDevice<bool> configured;
  if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
  int units = tiles * p.splits;
  if (units > num_sms / 2) units = num_sms / 2;
  const bool early = p.K <= 32768;                         // as in launch()
  launch_early_if(early, kern, 2 * units, kThreads, C::kTotal, stream, 0, maps[0], maps[1], p);
  return cudaGetLastError();
}

// clusters of `splits` blocks that run at a time: one block per SM, so the same for all forms of the operands, whose blocks are alike
static_assert(Cfg<1, 64, true>::kTotal == Cfg<1, 64, false>::kTotal && Cfg<1, 128, true>::kTotal == Cfg<1, 128, false>::kTotal && Cfg<1, 64>::kTotal > kSmemBudget / 2 &&
              Cfg<1, 128>::kTotal > kSmemBudget / 2, "auto_splits asks for one form");
template <int BN, bool A_MN, bool B_MN>
static int splitk_clusters(int splits) {
  using C = Cfg<1, BN, B_MN>;
  if (splits < 2 || splits > kMaxClusterSplits) return 0;
  static nrl::PerDevice<ClusterCounts> counts;
  return clusters_of(counts, gemm_tc_splitk_cluster_kernel<BN, A_MN, B_MN>, C::kTotal, splits);
}

template <int BN, bool A_MN, bool B_MN>
static cudaError_t launch_splitk(const CUtensorMap* maps, const TcParams& p, int num_sms, cudaStream_t stream) {
  using C = Cfg<1, BN, B_MN>;
  const int tiles = ((p.M + BLOCK_M - 1) / BLOCK_M) * ((p.N + BN - 1) / BN);
  int grid = tiles * p.splits;
  if (grid <= num_sms && split_by_clusters(p.splits, (p.K + BLOCK_K - 1) / BLOCK_K) && tiles <= splitk_clusters<BN, A_MN, B_MN>(p.splits)) {
    launch_dependent_clusters(gemm_tc_splitk_cluster_kernel<BN, A_MN, B_MN>, grid, kThreads, C::kTotal, stream, p.splits, maps[0], maps[1], p);
    return cudaGetLastError();
  }
  auto kern = gemm_tc_splitk_kernel<BN, A_MN, B_MN>;
  static nrl::PerDevice<bool> configured;
  if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
  if (grid > num_sms) grid = num_sms;
  launch_dependent(kern, grid, kThreads, C::kTotal, stream, maps[0], maps[1], p);
  return cudaGetLastError();
}

template <int CG, int BN, bool A_MN, bool B_MN, int EPI>
static cudaError_t launch(const CUtensorMap* maps, const TcParams& p, int num_sms, cudaStream_t stream) {
  using C = Cfg<CG, BN, B_MN>;
  const int num_m = (p.M + CG * BLOCK_M - 1) / (CG * BLOCK_M), num_n = (p.N + BN - 1) / BN;
  int units = num_m * (EPI == EPI_LOGPROB ? p.col_ranges : num_n);
  if (units > num_sms / CG) units = num_sms / CG;
  if (units < 1) units = 1;
  // Blocks that start early take the SMs that the kernel in front leaves first, side by side rather than spread over the chip, and share what those have of the way
  // to the L2: where there are fewer than SMs and the contraction is long that costs more than the start saves.  Log-probability head, 800 rows, forward and
  // backward (151 936 columns, 48 pairs of blocks) 1325 / 1309 us early / in order, 1000 rows 1470 / 1453, before overlapping launches 1310 / 1450; the line is
  // that of split_by_clusters, far from both sides' sizes (8960 columns, 18 to 74 pairs, gain).
  const bool early = p.K <= 32768;
  static nrl::PerDevice<bool> configured;
  if (CG == 1) {
    auto kern = gemm_tc_cg1_kernel<BN, A_MN, B_MN, EPI>;
    if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
    launch_early_if(early, kern, units, kThreads, C::kTotal, stream, 0, maps[0], maps[1], maps[2], maps[3], maps[4], p);
  } else {
    auto kern = gemm_tc_cg2_kernel<BN, A_MN, B_MN, EPI>;
    if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
    launch_early_if(early, kern, 2 * units, kThreads, C::kTotal, stream, 0, maps[0], maps[1], maps[2], maps[3], maps[4], p);   // consecutive CTAs pair up
  }
  return cudaGetLastError();
}

}  // namespace tc
}  // namespace nrl

extern "C" cudaError_t nrl_gemm_tc_dlogits(const CUtensorMap* maps, const nrl::tc::TcParams* p, int num_sms, cudaStream_t stream) {
  const CUtensorMap all[5] = {maps[0], maps[1], maps[0], maps[1], maps[2]};
  return nrl::tc::launch<2, 256, false, false, nrl::tc::EPI_DLOGITS>(all, *p, num_sms, stream);
}

// e4m3 x e4m3 GEMM with per-row x per-column scales; maps = {A (uint8 [M,K], box {128, 128}), B (uint8 [N,K], box {bn/cg, 128}), D}
extern "C" cudaError_t nrl_gemm_tc_fp8(const CUtensorMap* maps, const nrl::tc::TcParams* p, int cg, int bn, int swiglu, int num_sms,
                                       cudaStream_t stream) {
  using namespace nrl::tc;
  if (p->row_scale == nullptr || p->col_scale == nullptr || p->K2 != 0) return cudaErrorInvalidValue;
#define NRL_TC_FP8(CG_, BN_)                                                                                     \
  if (cg == CG_ && bn == BN_)                                                                                    \
    return swiglu ? launch_fp8<CG_, BN_, EPI_SWIGLU>(maps, *p, num_sms, stream) : launch_fp8<CG_, BN_, EPI_BF16>(maps, *p, num_sms, stream);
  NRL_TC_FP8(1, 128)
  NRL_TC_FP8(1, 256)
  NRL_TC_FP8(2, 128)
  NRL_TC_FP8(2, 256)
#undef NRL_TC_FP8
  if (!swiglu && cg == 2 && bn == 192) return launch_fp8<2, 192, EPI_BF16>(maps, *p, num_sms, stream);
  if (!swiglu && cg == 1 && bn == 192) return launch_fp8<1, 192, EPI_BF16>(maps, *p, num_sms, stream);
  return cudaErrorInvalidValue;
}

extern "C" cudaError_t nrl_gemm_tc_logprob(const CUtensorMap* maps, const nrl::tc::TcParams* p, int num_sms, cudaStream_t stream) {
  const CUtensorMap all[5] = {maps[0], maps[1], maps[0], maps[1], maps[0]};
  return nrl::tc::launch<2, 256, false, false, nrl::tc::EPI_LOGPROB>(all, *p, num_sms, stream);
}

template <int EPI>
static cudaError_t launch_pair(const CUtensorMap* maps, const nrl::tc::TcParams& p, int num_sms, cudaStream_t stream) {
  using namespace nrl::tc;
  using C = Cfg<2, 256, false>;
  auto kern = gemm_tc_pair_kernel<EPI>;
  static nrl::PerDevice<bool> configured;
  if (const cudaError_t e = nrl::allow_smem(configured, kern, C::kTotal); e != cudaSuccess) return e;
  int units = ((p.M + 255) / 256) * ((p.N + 255) / 256);
  if (units > num_sms / 2) units = num_sms / 2;
  if (units < 1) units = 1;
  TcMaps<EPI == EPI_SWIGLU_KEEP ? 3 : 1> more;
  more.m[0] = maps[4];
  if constexpr (EPI == EPI_SWIGLU_KEEP) {
    more.m[1] = maps[8];
    more.m[2] = maps[9];
  }
  nrl::launch_dependent(kern, 2 * units, kThreads, C::kTotal, stream, maps[0], maps[1], maps[2], maps[3], maps[5], maps[6], maps[7], more, p);
  return cudaGetLastError();
}
extern "C" cudaError_t nrl_gemm_tc_pair(const CUtensorMap* maps, const nrl::tc::TcParams* p, int keep, int num_sms, cudaStream_t stream) {
  if (p->N % 16 != 0) return cudaErrorInvalidValue;
  return keep ? launch_pair<nrl::tc::EPI_SWIGLU_KEEP>(maps, *p, num_sms, stream) : launch_pair<nrl::tc::EPI_SWIGLU>(maps, *p, num_sms, stream);
}

extern "C" cudaError_t nrl_gemm_tc_dswiglu(const CUtensorMap* maps, const nrl::tc::TcParams* p, int num_sms, cudaStream_t stream) {
  using namespace nrl::tc;
  using C = Cfg<2, 256, true, 2>;
  static nrl::PerDevice<bool> configured;
  if (const cudaError_t e = nrl::allow_smem(configured, gemm_tc_dswiglu_kernel, C::kTotal); e != cudaSuccess) return e;
  int units = ((p->M + 255) / 256) * ((p->N + 255) / 256);
  if (units > num_sms / 2) units = num_sms / 2;
  if (units < 1) units = 1;
  const TcMaps<3> more{{maps[4], maps[5], maps[7]}};
  nrl::launch_dependent(gemm_tc_dswiglu_kernel, 2 * units, kThreads, C::kTotal, stream, maps[0], maps[1], maps[2], maps[3], maps[6], more, *p);
  return cudaGetLastError();
}

extern "C" cudaError_t nrl_gemm_tc_sum(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int num_sms, cudaStream_t stream) {
  using namespace nrl::tc;
  TcMaps<2 * kSumPairs> all;
  for (int i = 0; i < 2 * kSumPairs; ++i) all.m[i] = maps[i];
  const CUtensorMap& d = maps[2 * kSumPairs];
  if (bn == 256) return launch_sum<256>(all, d, *p, num_sms, stream);
  if (bn == 192) return launch_sum<192>(all, d, *p, num_sms, stream);
  if (bn == 128) return launch_sum<128>(all, d, *p, num_sms, stream);
  return cudaErrorInvalidValue;
}

extern "C" cudaError_t nrl_gemm_tc_cat(const CUtensorMap* maps, const nrl::tc::TcParams* p, const nrl::tc::TcCat* cat, int cg, int bn, int num_sms, cudaStream_t stream) {
  using namespace nrl::tc;
  TcMaps<4 * kCatMax> all;
  for (int i = 0; i < 4 * kCatMax; ++i) all.m[i] = maps[1 + i];
#define NRL_TC_CAT(CG_, BN_) \
  if (cg == CG_ && bn == BN_) return launch_cat<CG_, BN_>(maps[0], all, *p, *cat, num_sms, stream);
  NRL_TC_CAT(1, 64) NRL_TC_CAT(1, 128) NRL_TC_CAT(2, 128) NRL_TC_CAT(2, 192) NRL_TC_CAT(2, 256)
#undef NRL_TC_CAT
  return cudaErrorInvalidValue;
}

extern "C" cudaError_t nrl_gemm_tc_batched(const CUtensorMap* maps, const nrl::tc::TcParams* p, int cg, int bn, int num_sms,
                                           cudaStream_t stream) {
  using namespace nrl::tc;
  if (p->batch < 1 || p->K2 != 0) return cudaErrorInvalidValue;
  if (cg == 1 && bn == 128) return launch_batched<1, 128>(maps, *p, num_sms, stream);
  if (cg == 1 && bn == 256) return launch_batched<1, 256>(maps, *p, num_sms, stream);
  if (cg == 2 && bn == 128) return launch_batched<2, 128>(maps, *p, num_sms, stream);
  if (cg == 2 && bn == 256) return launch_batched<2, 256>(maps, *p, num_sms, stream);
  return cudaErrorInvalidValue;
}

extern "C" cudaError_t nrl_gemm_tc_grouped(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int max_tiles, int num_sms,
                                           cudaStream_t stream) {
  using namespace nrl::tc;
  if (p->grp_tiles == nullptr || p->grp_num_tiles == nullptr || p->K2 != 0 || max_tiles < 1 || p->N % 4 != 0) return cudaErrorInvalidValue;
  if (p->out_bf16 == nullptr ? p->out_f32 == nullptr : (p->N % (p->act == 2 ? 8 : 64) != 0 || p->out_stride % 8 != 0)) return cudaErrorInvalidValue;
  if (bn == 64) return launch_grouped<64>(maps, *p, max_tiles, num_sms, stream);
  if (bn == 128) return launch_grouped<128>(maps, *p, max_tiles, num_sms, stream);
  if (bn == 256) return launch_grouped<256>(maps, *p, max_tiles, num_sms, stream);
  return cudaErrorInvalidValue;
}

extern "C" int nrl_gemm_tc_multi_clusters(int a_mn, int splits) {
  return a_mn ? nrl::tc::multi_clusters<true, true>(splits) : nrl::tc::multi_clusters<false, true>(splits);
}
extern "C" cudaError_t nrl_gemm_tc_multi(const CUtensorMap* maps, const nrl::tc::TcMultiProduct* products, int n, int a_mn, int splits, cudaStream_t stream) {
  using namespace nrl::tc;
  if (n < 1 || n > kMultiMax || splits < 1) return cudaErrorInvalidValue;
  TcMulti m;
  int tiles = 0;
  for (int i = 0; i < n; ++i) {
    const TcMultiProduct& q = products[i];
    if (q.M < 1 || q.N < 1 || q.K < 1 || q.out == nullptr) return cudaErrorInvalidValue;
    tiles += ((q.M + BLOCK_M - 1) / BLOCK_M) * ((q.N + 63) / 64);
    m.a[i] = maps[2 * i];
    m.b[i] = maps[2 * i + 1];
    m.tiles[i] = tiles;
    m.M[i] = q.M; m.N[i] = q.N; m.K[i] = q.K;
    m.alpha[i] = q.alpha;
    m.out[i] = static_cast<__nv_bfloat16*>(q.out);
    m.stride[i] = q.stride;
    m.transposed[i] = q.transposed;
  }
  return a_mn ? launch_multi<true, true>(m, n, splits, stream) : launch_multi<false, true>(m, n, splits, stream);
}

extern "C" int nrl_gemm_tc_pair_clusters(int bn, int splits) {
  using namespace nrl::tc;
  return bn == 128 ? split_pairs_clusters<128, false>(splits) : bn == 192 ? split_pairs_clusters<192, false>(splits) : split_pairs_clusters<256, false>(splits);
}
extern "C" cudaError_t nrl_gemm_tc_split_pairs(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int b_mn, int clusters, int num_sms,
                                               cudaStream_t stream) {
  using namespace nrl::tc;
  if (p->splits < 2 || p->out_bf16 == nullptr || p->K2 != 0) return cudaErrorInvalidValue;
#define NRL_TC_PAIRS(BN_, BMN_) \
  if (bn == BN_ && b_mn == (BMN_ ? 1 : 0)) return launch_split_pairs<BN_, BMN_>(maps, *p, clusters != 0, num_sms, stream);
  NRL_TC_PAIRS(128, false)
  NRL_TC_PAIRS(128, true)
  NRL_TC_PAIRS(192, false)
  NRL_TC_PAIRS(192, true)
  NRL_TC_PAIRS(256, false)
  NRL_TC_PAIRS(256, true)
#undef NRL_TC_PAIRS
  return cudaErrorInvalidValue;
}

extern "C" int nrl_gemm_tc_split_clusters(int bn, int splits) {
  return bn == 64 ? nrl::tc::splitk_clusters<64, false, false>(splits) : nrl::tc::splitk_clusters<128, false, false>(splits);
}

// split-K variant (cta_group::1, bf16 output with plain stores, no second operand pair); maps = {A, B}
extern "C" cudaError_t nrl_gemm_tc_splitk(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int a_mn, int b_mn, int num_sms,
                                          cudaStream_t stream) {
  using namespace nrl::tc;
  if (p->splits < 1 || p->ws == nullptr || p->counters == nullptr || p->out_bf16 == nullptr || p->K2 != 0) return cudaErrorInvalidValue;
#define NRL_TC_SPLIT(BN_, AMN_, BMN_) \
  if (bn == BN_ && a_mn == (AMN_ ? 1 : 0) && b_mn == (BMN_ ? 1 : 0)) return launch_splitk<BN_, AMN_, BMN_>(maps, *p, num_sms, stream);
  NRL_TC_SPLIT(64, false, false)
  NRL_TC_SPLIT(128, false, false)
  NRL_TC_SPLIT(64, false, true)
  NRL_TC_SPLIT(128, false, true)
  NRL_TC_SPLIT(64, true, true)
  NRL_TC_SPLIT(128, true, true)
#undef NRL_TC_SPLIT
  return cudaErrorInvalidValue;
}

// maps = {A, B, A2, B2, D}; operand boxes (tma_host.h): K-major operand [rows, K]: box {rows = 128 (A) | BN/CG (B), 64};
// MN-major operand [K, cols]: box {64, 64}; D: box {32, 64}.  Unused maps may repeat a valid one.
extern "C" cudaError_t nrl_gemm_tc(const CUtensorMap* maps, const nrl::tc::TcParams* p, int cg, int bn, int a_mn, int b_mn,
                                   int epi, int num_sms, cudaStream_t stream) {
  using namespace nrl::tc;
#define NRL_TC_CASE(CG_, BN_, AMN_, BMN_, EPI_)                                                             \
  if (cg == CG_ && bn == BN_ && a_mn == (AMN_ ? 1 : 0) && b_mn == (BMN_ ? 1 : 0) && epi == EPI_)             \
    return launch<CG_, BN_, AMN_, BMN_, EPI_>(maps, *p, num_sms, stream);
  // K-major x K-major ("TN": forward linears, LoRA down-projection, DeBERTa)
  NRL_TC_CASE(1, 64, false, false, EPI_BF16)
  NRL_TC_CASE(1, 128, false, false, EPI_BF16)
  NRL_TC_CASE(1, 192, false, false, EPI_BF16)
  NRL_TC_CASE(1, 256, false, false, EPI_BF16)
  NRL_TC_CASE(2, 128, false, false, EPI_BF16)
  NRL_TC_CASE(2, 192, false, false, EPI_BF16)
  NRL_TC_CASE(2, 256, false, false, EPI_BF16)
  NRL_TC_CASE(1, 64, false, false, EPI_RESIDUAL)
  NRL_TC_CASE(1, 128, false, false, EPI_RESIDUAL)
  NRL_TC_CASE(1, 192, false, false, EPI_RESIDUAL)
  NRL_TC_CASE(1, 256, false, false, EPI_RESIDUAL)
  NRL_TC_CASE(2, 128, false, false, EPI_RESIDUAL)
  NRL_TC_CASE(2, 192, false, false, EPI_RESIDUAL)
  NRL_TC_CASE(2, 256, false, false, EPI_RESIDUAL)
  NRL_TC_CASE(1, 128, false, false, EPI_SWIGLU)
  NRL_TC_CASE(1, 256, false, false, EPI_SWIGLU)
  NRL_TC_CASE(2, 128, false, false, EPI_SWIGLU)
  NRL_TC_CASE(2, 256, false, false, EPI_SWIGLU)
  // K-major x MN-major ("NN": dgrad  dX = dY W, dH = dZ W_lm)
  NRL_TC_CASE(1, 64, false, true, EPI_BF16)
  NRL_TC_CASE(1, 128, false, true, EPI_BF16)
  NRL_TC_CASE(1, 192, false, true, EPI_BF16)
  NRL_TC_CASE(1, 256, false, true, EPI_BF16)
  NRL_TC_CASE(2, 128, false, true, EPI_BF16)
  NRL_TC_CASE(2, 192, false, true, EPI_BF16)
  NRL_TC_CASE(2, 256, false, true, EPI_BF16)
  // MN-major x MN-major ("NT": wgrad  dW = dY^T X)
  NRL_TC_CASE(1, 64, true, true, EPI_BF16)
  NRL_TC_CASE(1, 128, true, true, EPI_BF16)
  NRL_TC_CASE(1, 256, true, true, EPI_BF16)
  NRL_TC_CASE(2, 256, true, true, EPI_BF16)
  NRL_TC_CASE(1, 64, true, true, EPI_F32)
  NRL_TC_CASE(1, 128, true, true, EPI_F32)
  NRL_TC_CASE(1, 256, true, true, EPI_F32)
  NRL_TC_CASE(2, 256, true, true, EPI_F32)
  // K-major x K-major with the float32 epilogue (hybrid decoders: projections feeding float32 recurrences / the residual)
  NRL_TC_CASE(1, 64, false, false, EPI_F32)
  NRL_TC_CASE(1, 128, false, false, EPI_F32)
  NRL_TC_CASE(1, 256, false, false, EPI_F32)
  NRL_TC_CASE(2, 256, false, false, EPI_F32)
#undef NRL_TC_CASE
  return cudaErrorInvalidValue;
}
