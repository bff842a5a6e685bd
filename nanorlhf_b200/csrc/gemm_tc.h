// Host-visible parameter block of the general tcgen05 GEMM (gemm_tc.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace nrl {
namespace tc {

enum TcEpilogue : int {
  EPI_BF16 = 0,      // D (bf16, TMA store) = alpha * acc (+ bias) (GELU)
  EPI_F32 = 1,       // out_f32 (row-major, plain stores) (+)= alpha * acc
  EPI_DLOGITS = 3,   // D (bf16, TMA store) = (onehot(target) - exp(alpha * acc - lse)) * grad * alpha: backward of the log-prob head
  EPI_GRP_SWIGLU = 4,  // GROUPED: out_bf16 [rows, N / 2] = silu(gate) * up of row_scale * acc, B rows interleaved as for EPI_SWIGLU, plain stores
  EPI_GRP_RELU2 = 5,   // GROUPED: out_bf16 [rows, N] = relu(row_scale * acc)^2, plain stores
  EPI_SWIGLU_KEEP = 6,  // PAIR kernels: as EPI_SWIGLU, and gate and up (bf16, TMA store)
  EPI_DSWIGLU = 7,   // D, D2 (bf16, TMA store) = gradients of gate and up, acc being that of silu(gate) * up
  EPI_LOGPROB = 8,   // out_f32 [2 col_ranges, M, 4] = statistics of a row over half a range's columns: max, sum of exp, sum of exp * logit, target's logit
  EPI_RESIDUAL = 9,  // EPI_BF16 and a residual [M, N] added to the rounded result, K-major operands
  EPI_SWIGLU = 2,    // D[M, N/2] (bf16, TMA store) = silu(gate) * up; B rows interleaved per 32 features [32 gate | 32 up]
};

constexpr int kSumPairs = 4;    // products that one accumulator takes (nrl_gemm_tc_sum)
constexpr int kMultiMax = 6;    // products of one launch (nrl_gemm_tc_multi)
struct TcMultiProduct {         // out [M, N] (row stride `stride`) or, transposed, [N, M] = alpha A B
  int M, N, K;
  float alpha;
  void* out;
  long stride;
  int transposed;
};

constexpr int kCatMax = 4;      // products of one input side by side (nrl_gemm_tc_cat)
struct TcCat {
  int end[kCatMax];             // column tiles of the products up to and with the i-th (of those behind the last: as many)
  int n[kCatMax];               // its columns
  const __nv_bfloat16* bias[kCatMax];
};

struct TcParams {
  int M, N, K;                  // D is [M, N]; K = contraction length of the first operand pair
  int K2;                       // contraction length of the second operand pair (0 = none)
  // of one kernel at most; the parameters travel with every launch
  union {
    struct {
      const float* row_scale;   // FP8 kernels: [M] per-token dequantisation scale of A (GROUPED: see below)
      const float* col_scale;   // FP8 kernels: [N] per-output-channel dequantisation scale of B
    };
    struct {
      const __nv_bfloat16* residual;      // EPI_RESIDUAL: [M, N], row stride residual_stride
      long residual_stride;
    };
    float* logits;              // EPI_LOGPROB: null, or [M, N] for the accumulator
    int sum_end[kSumPairs];     // SUM kernels: k-blocks of the products up to and with the i-th (of those behind the last: as many)
  };
  const int* targets;           // EPI_LOGPROB, EPI_DLOGITS: [M] column of the row's target
  const float* lse;             // EPI_DLOGITS: [M] log of the row's sum of exponentials
  const float* grad;            // EPI_DLOGITS: [M] gradient of the row's log-probability
  int batch;                    // BATCH kernels: number of independent [M,K] x [N,K]^T problems behind 3D tensor maps (else 1)
  float alpha;                  // multiplies the accumulator
  const __nv_bfloat16* bias;    // EPI_BF16: optional [N]
  union {
    int act;                    // EPI_BF16: 0 = none, 1 = exact (erf) GELU after the bias (GROUPED: see below)
    int col_ranges;             // EPI_LOGPROB: into how many ranges the column tiles are cut (work items = row tiles x ranges)
  };
  float* out_f32;               // EPI_F32: [M, N] fp32, row stride out_f32_stride elements
  long out_f32_stride;
  union {
    int accumulate;             // EPI_F32: 1 = add to what is there
    int transposed;             // MULTI kernels: D^T [N, M] is written
  };
  // split-K (SPLIT kernels; small outputs with a long contraction -- LoRA wgrads, rank-r projections): every tile is
  // computed by `splits` CTAs over disjoint k-ranges; where they fit they are a cluster that sums its partial tiles through distributed shared memory,
  // else partial tiles go to `ws` (fp32) and the last CTA to arrive on the tile's counter sums them.  Either way in split order
  // (deterministic), bf16 result.  Counters reset themselves.
  int splits;
  float* ws;                    // [splits, tiles, 128, BN] fp32
  int* counters;                // [tiles] int32, zero between launches
  __nv_bfloat16* out_bf16;      // SPLIT: D written with plain stores (row stride out_stride elements)
  long out_stride;
  // GROUPED kernels (mixture of experts): the rows of A are sorted by expert and B holds every expert's [N, K] matrix one after
  // the other.  A row tile belongs to one expert; it may start at any row and is cut off at the end of the expert's rows
  // (the tile's further rows are computed and dropped).  The table and its length live on the device (written by the
  // routing kernels of the same stream), so no launch parameter depends on the routing.
  const int* grp_tiles;         // [max tiles, 3]: expert, first row, end row (exclusive) of the expert's rows
  const int* grp_num_tiles;     // [1]: row tiles in use
};

// 56 bytes more made four projections in a row 0.4 of 43 us slower (39 and 81 rows; in a graph as fast): the device reads them launch by launch
static_assert(sizeof(TcParams) <= 152, "launch parameters of every GEMM");

// Is a contraction of `blocks` times 64 columns in `splits` ranges summed by clusters (where they fit)?  Not two long ranges: a cluster of two takes both SMs of a
// pair that share their way to the L2 and leaves other pairs idle, which costs more than the sum through the workspace from 32 768 columns on.  us, clusters /
// workspace: 400 x 1536 over 32 768 columns 67.0 / 66.9, 65 536 127.5 / 118.2, 151 936 272 / 263; 554 x 1536 over 16 384 35.7 / 36.8, 32 768 66.7 / 67.1, 65 536 128.6 /
// 126.9, 151 936 296 / 290; three ranges of 300 x 1536 over 65 536 85.3 / 85.5, eight of 100 x 1536 41.5 / 48.4.
inline bool split_by_clusters(int splits, long blocks) { return splits > 2 || blocks <= 512; }

}  // namespace tc
}  // namespace nrl

// n products in one launch, B MN-major [K, N] (box {64, 64}), A MN-major [K, M] (a_mn, box {64, 64}) or K-major [M, K] (box {128, 64}); maps = {A_0, B_0, A_1 ..}; bf16
// results with plain stores, N and, transposed, the stride multiples of 8; every contraction cut into `splits` ranges, none empty, summed by clusters
extern "C" int nrl_gemm_tc_multi_clusters(int a_mn, int splits);
extern "C" cudaError_t nrl_gemm_tc_multi(const CUtensorMap* maps, const nrl::tc::TcMultiProduct* products, int n, int a_mn, int splits, cudaStream_t stream);
// clusters of `splits` blocks that run at a time (0: none), whichever form the operands have
extern "C" int nrl_gemm_tc_split_clusters(int bn, int splits);
// the same for clusters of `splits` pairs of blocks (tiles of 256 x bn), and the GEMM that they run: A K-major (box {128, 64}), B box {bn / 2, 64} or, MN-major,
// {64, 64}; bf16 output with plain stores; p->splits ranges, none empty
extern "C" int nrl_gemm_tc_pair_clusters(int bn, int splits);
extern "C" cudaError_t nrl_gemm_tc_split_pairs(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int b_mn, int clusters, int num_sms,
                                               cudaStream_t stream);
extern "C" cudaError_t nrl_gemm_tc_splitk(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int a_mn, int b_mn, int num_sms,
                                          cudaStream_t stream);
// EPI_DLOGITS on CTA pairs, 256 x 256 tiles; maps = {A box {128, 64}, B box {128, 64}, D box {32, 64}}
extern "C" cudaError_t nrl_gemm_tc_dlogits(const CUtensorMap* maps, const nrl::tc::TcParams* p, int num_sms, cudaStream_t stream);
// EPI_LOGPROB likewise; maps = {A box {128, 64}, B box {128, 64}}
extern "C" cudaError_t nrl_gemm_tc_logprob(const CUtensorMap* maps, const nrl::tc::TcParams* p, int num_sms, cudaStream_t stream);
extern "C" cudaError_t nrl_gemm_tc_fp8(const CUtensorMap* maps, const nrl::tc::TcParams* p, int cg, int bn, int swiglu, int num_sms,
                                       cudaStream_t stream);
// batched K-major x K-major GEMM, bf16 out; maps = {A, B, D} 3D (tma_host.h make_tma_3d), B box rows = bn / cg
extern "C" cudaError_t nrl_gemm_tc_batched(const CUtensorMap* maps, const nrl::tc::TcParams* p, int cg, int bn, int num_sms,
                                           cudaStream_t stream);
// grouped K-major x K-major GEMM (cta_group 1); maps = {A [rows, K] box {128, 64}, B [experts * N, K] box {bn, 64}};
// p->N = columns per expert; max_tiles bounds the table's length (grid size).  Output: out_f32 [rows, N], or, when out_bf16 is
// set, the SwiGLU of the columns: B rows interleaved per 32 features ([32 gate | 32 up], N % 64 == 0), out_bf16 [rows, N / 2]
// (row stride out_stride, a multiple of 8) = silu(gate) * up; row_scale [rows] (or null) then multiplies gate and up first.  act == 2: the
// squared ReLU of the columns instead, out_bf16 [rows, N] = relu(row_scale * x)^2, B rows in their own order.
extern "C" cudaError_t nrl_gemm_tc_grouped(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int max_tiles, int num_sms,
                                           cudaStream_t stream);
// act [M, F] = silu(x Wg^T + tg Bg^T) * (x Wu^T + tu Bu^T); maps = {x box {128, 64}, Wg, Wu box {128, 64}, tg, tu box {128, 64}, Bg, Bu box
// {128, 64}, act box {32, 64}}; p->N = 2 F, p->K2 = columns of tg and tu (0: no adapters, maps 3 .. 6 may repeat a valid one); keep: x Wg^T + tg Bg^T
// and x Wu^T + tu Bu^T too, through maps 8 and 9, box {32, 64}
extern "C" cudaError_t nrl_gemm_tc_pair(const CUtensorMap* maps, const nrl::tc::TcParams* p, int keep, int num_sms, cudaStream_t stream);
// gradients of gate and up [M, N] from dY [M, K], W [K, N], T [M, K2], A [K2, N] (K2 may be 0): maps = {dY box {128, 64}, W box {64, 64}, T box {128, 64},
// A box {64, 64}, gate, up, d gate, d up, box {32, 64}}
extern "C" cudaError_t nrl_gemm_tc_dswiglu(const CUtensorMap* maps, const nrl::tc::TcParams* p, int num_sms, cudaStream_t stream);
// D_i = x W_i^T + T_i B_i^T (+ bias_i) for up to kCatMax i with one x and equal K and K2; maps = {x box {128, 64}, then kCatMax each of W box {bn / cg, 64},
// T box {128, 64}, B box {bn / cg, 64}, D box {32, 64}}
extern "C" cudaError_t nrl_gemm_tc_cat(const CUtensorMap* maps, const nrl::tc::TcParams* p, const nrl::tc::TcCat* cat, int cg, int bn, int num_sms, cudaStream_t stream);
// D [M, N] = sum of A_i [M, K_i] B_i [K_i, N] on CTA pairs; maps = {A_0 .. A_3 box {128, 64}, B_0 .. B_3 box {64, 64}, D box {32, 64}}, unused ones repeat a
// valid one; p->sum_end as there
extern "C" cudaError_t nrl_gemm_tc_sum(const CUtensorMap* maps, const nrl::tc::TcParams* p, int bn, int num_sms, cudaStream_t stream);
extern "C" cudaError_t nrl_gemm_tc(const CUtensorMap* maps, const nrl::tc::TcParams* p, int cg, int bn, int a_mn, int b_mn,
                                   int epi, int num_sms, cudaStream_t stream);
