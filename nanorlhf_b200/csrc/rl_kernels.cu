// RL-specific fused kernels:
//   K-GAE  gae_scan          reverse linear-recurrence scan (GAE / discounted suffix sums), block per sequence
//   K-LOSS policy_loss       PPO-clip (+ GRPO k3-KL) forward + gradient + all statistics in ONE pass
//          value_loss        clipped value loss forward + gradient
//   K18    adamw_flat        AdamW over flat bf16 parameter / gradient buffers with fp32 or bf16 moments
// Reference: the python time-step loop (GRPO/grpo_trainer.py:611-617, PPO/ppo_trainer.py:
// 688-697), ~15 elementwise launches per micro-batch (:662-688) and torch AdamW (:692).
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace nrl {

// ---- K-GAE ------------------------------------------------------------------------------------
// A_t = delta_t + c * A_{t+1},  delta_t = r_t + gamma * V_{t+1} - V_t  (V == nullptr -> delta = r, c = gamma*lam)
// Block per row, kGaePer consecutive steps per thread: a thread folds its own steps, a weighted reverse scan over the warp and one over
// the warps give every thread the advantage behind its last step, and the recurrence is then run as it is written.  4 x 1500 steps: 15 us
// with one warp per row (47 dependent rounds of load and shuffle), 3.6 us here; longer rows go tile by tile from the end.  In double: powers of
// a rounded c cost more than the sums themselves (error against float64 2.4e-7 -> 2.5e-8).
// Rows that one warp holds (256 steps) take a warp each, four to a block, without barriers: 512 x 100 steps 2.6 us, a block per row 4.1; one row of 64
// 2.5 us either way.
constexpr int kGaeWarps = 8, kGaePer = 8, kGaeRows = 4;

template <int WARPS>                                  // that share a row: kGaeWarps, or 1 and kGaeRows rows to a block
__global__ void __launch_bounds__(32 * (WARPS == 1 ? kGaeRows : WARPS))
gae_scan_kernel(const float* __restrict__ rewards, const float* __restrict__ values, float* __restrict__ adv,
                float* __restrict__ returns, int B, int T, double gamma, double lam) {
  constexpr int kTile = 32 * WARPS * kGaePer;
  __shared__ double heads[WARPS + 1];                 // folded value of every warp's steps; one more: the tile's first advantage
  const int lane = threadIdx.x & 31, warp = WARPS == 1 ? 0 : threadIdx.x >> 5, tid = warp * 32 + lane;
  const int seq = WARPS == 1 ? blockIdx.x * kGaeRows + (threadIdx.x >> 5) : blockIdx.x;
  if (seq >= B) return;
  const size_t row = static_cast<size_t>(seq) * T;
  const float* r = rewards + row;
  const float* v = values ? values + row : nullptr;
  const double c = gamma * lam;
  double w[6];                                       // c^8, c^16 .. c^256: weights of a step of the scan
  w[0] = c * c;
  w[0] *= w[0];
  w[0] *= w[0];
#pragma unroll
  for (int k = 1; k < 6; ++k) w[k] = w[k - 1] * w[k - 1];
  double c_lane = 1.0;                                // c^(8 * (32 - lane - 1)): from the next warp's first step to this thread's last
#pragma unroll
  for (int k = 0; k < 5; ++k)
    if ((31 - lane) & (1 << k)) c_lane *= w[k];
  double behind = 0.0;                                // advantage of the step behind the tile
  for (int tile = (T - 1) / kTile; tile >= 0; --tile) {
    const int t0 = tile * kTile + tid * kGaePer;
    double d[kGaePer];
    float vt[kGaePer];
#pragma unroll
    for (int j = 0; j < kGaePer; ++j) {
      d[j] = t0 + j < T ? r[t0 + j] : 0.0;
      vt[j] = v != nullptr && t0 + j < T ? v[t0 + j] : 0.f;
    }
    if (v != nullptr) {
      const float vn = t0 + kGaePer < T ? v[t0 + kGaePer] : 0.f;
#pragma unroll
      for (int j = 0; j < kGaePer; ++j) d[j] += gamma * (j + 1 < kGaePer ? vt[j + 1] : vn) - vt[j];
    }
    double x = 0.0;
#pragma unroll
    for (int j = kGaePer - 1; j >= 0; --j) x = fma(c, x, d[j]);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const double y = __shfl_down_sync(0xffffffffu, x, 1 << k);
      if (lane + (1 << k) < 32) x = fma(w[k], y, x);
    }
    double in = behind;                               // advantage at the first step of the next warp
    if (WARPS > 1) {
      __syncthreads();                               // `heads` of the tile before has been read
      if (lane == 0) heads[warp] = x;
      __syncthreads();
      for (int q = WARPS - 1; q > warp; --q) in = fma(w[5], in, heads[q]);
    }
    const double next = __shfl_down_sync(0xffffffffu, x, 1);
    double a = fma(c_lane, in, lane < 31 ? next : 0.0);
#pragma unroll
    for (int j = kGaePer - 1; j >= 0; --j) {
      a = fma(c, a, d[j]);
      if (t0 + j < T) {
        adv[row + t0 + j] = static_cast<float>(a);
        if (returns) returns[row + t0 + j] = static_cast<float>(a + vt[j]);
      }
    }
    if (WARPS > 1) {
      if (tid == 0) heads[WARPS] = a;
      __syncthreads();
      behind = heads[WARPS];
    } else {
      behind = __shfl_sync(0xffffffffu, a, 0);
    }
  }
}

// ---- K-LOSS -----------------------------------------------------------------------------------
// Sums over all tokens in double (masked losses cancel) and in a fixed order, finished inside the launch: up to kLossClusterMax tokens the blocks are one cluster and leave
// their sums in the first block's shared memory; above, they leave them in `scratch` and the block that arrives last adds them up.
// Every quotient of sums was a launch of its own before: 28 launches, 58 us of kernels and 342 us in all for the losses and advantages of a PPO
// micro-step of 4 x 1500 tokens; 11 launches, 24 us of kernels and about 160 us in all with these.
constexpr int kLossThreads = 512;
constexpr long kLossClusterMax = 1 << 17;
constexpr unsigned kLossBlocks = 148;               // a number of its own, so that the order of the sums does not depend on the device

// A block's shared memory may be written by the others of its cluster once it is known to run: every thread arrives on entry to the kernel and
// waits in front of the first remote write, so that the pass over the tokens hides the barrier.
__device__ __forceinline__ void cluster_started_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_started_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

template <int NS>
__device__ bool loss_sums(double (&s)[NS], double* scratch, double (&tot)[NS]) {      // true in the one thread that has the totals
  namespace cg = cooperative_groups;
  __shared__ double red[NS][kLossThreads / 32];
  __shared__ double parts[8][NS];
  __shared__ int last;
#pragma unroll
  for (int j = 0; j < NS; ++j) s[j] = warp_sum(s[j]);
  if (lane_id() == 0)
#pragma unroll
    for (int j = 0; j < NS; ++j) red[j][threadIdx.x >> 5] = s[j];
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < NS)
    for (int q = 0; q < kLossThreads / 32; ++q) t += red[threadIdx.x][q];
  if (scratch == nullptr) {
    cg::cluster_group cl = cg::this_cluster();
    cluster_started_wait();
    if (threadIdx.x < NS) cl.map_shared_rank(&parts[0][0], 0)[cl.block_rank() * NS + threadIdx.x] = t;
    cl.sync();
    if (cl.block_rank() != 0 || threadIdx.x != 0) return false;
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      tot[j] = 0.0;
      for (unsigned q = 0; q < cl.num_blocks(); ++q) tot[j] += parts[q][j];
    }
    return true;
  }
  int* counter = reinterpret_cast<int*>(scratch);
  double* slots = scratch + 1;
  if (threadIdx.x < NS) slots[blockIdx.x * NS + threadIdx.x] = t;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1) == static_cast<int>(gridDim.x) - 1;
  __syncthreads();
  if (!last || threadIdx.x != 0) return false;
  __threadfence();
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    tot[j] = 0.0;
    for (unsigned q = 0; q < gridDim.x; ++q) tot[j] += __ldcg(slots + q * NS + j);
  }
  return true;
}

// grad_unnorm[i] = d(per-token loss)/d(new_logp) * m   (the backward divides by sum(m)).  loss[0]; stats: sum(m), clip fraction, 0.5 mean
// diff^2 over masked / all tokens, mean ratio over all / masked tokens, mean k over all / masked tokens
__global__ void __launch_bounds__(kLossThreads)
policy_loss_kernel(const float* __restrict__ new_lp, const float* __restrict__ old_lp, const float* __restrict__ adv,
                   const uint8_t* __restrict__ mask, const float* __restrict__ ref_lp, float cliprange, float kl_coef, long n,
                   float* __restrict__ grad_unnorm, float* __restrict__ loss, float* __restrict__ stats, double* scratch) {
  if (scratch == nullptr) cluster_started_arrive();
  double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float nl = new_lp[i], ol = old_lp[i], a = adv[i];
    const float m = mask[i] ? 1.f : 0.f;
    const float diff = nl - ol;
    const float ratio = __expf(diff);
    const float l1 = -a * ratio;
    const float rc = fminf(fmaxf(ratio, 1.f - cliprange), 1.f + cliprange);
    const float l2 = -a * rc;
    float per = fmaxf(l1, l2);
    // d max(l1,l2)/d nl: l1 branch -> -a*ratio ; l2 branch -> 0 when clipped, -a*ratio when not clipped
    const bool clipped_active = (l2 > l1);
    float g = clipped_active ? ((rc == ratio) ? -a * ratio : 0.f) : -a * ratio;
    float k = 0.f;
    if (ref_lp != nullptr) {
      k = nl - ref_lp[i];
      const float e = __expf(-k);
      per += kl_coef * (e + k - 1.f);
      g += kl_coef * (1.f - e);
    }
    grad_unnorm[i] = g * m;
    s[0] += per * m; s[1] += m; s[2] += clipped_active ? m : 0.f;
    s[3] += diff * diff * m; s[4] += diff * diff; s[5] += ratio; s[6] += ratio * m; s[7] += k; s[8] += k * m;
  }
  double t[9];
  if (!loss_sums(s, scratch, t)) return;
  const double all = static_cast<double>(n);
  loss[0] = static_cast<float>(t[0] / t[1]);
  stats[0] = static_cast<float>(t[1]);
  stats[1] = static_cast<float>(t[2] / t[1]);
  stats[2] = static_cast<float>(0.5 * t[3] / t[1]);
  stats[3] = static_cast<float>(0.5 * t[4] / all);
  stats[4] = static_cast<float>(t[5] / all);
  stats[5] = static_cast<float>(t[6] / t[1]);
  stats[6] = static_cast<float>(t[7] / all);
  stats[7] = static_cast<float>(t[8] / t[1]);
}

// loss[0] = 0.5 sum(max(l1,l2)*m) / sum(m); stats: sum(m), share of masked tokens with l2 > l1; grad_unnorm = d(0.5*max)/d vpred * m
__global__ void __launch_bounds__(kLossThreads)
value_loss_kernel(const float* __restrict__ vpred, const float* __restrict__ vold, const float* __restrict__ ret,
                  const uint8_t* __restrict__ mask, float clip, long n, float* __restrict__ grad_unnorm, float* __restrict__ loss,
                  float* __restrict__ stats, double* scratch) {
  if (scratch == nullptr) cluster_started_arrive();
  double s[3] = {0, 0, 0};
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float v = vpred[i], vo = vold[i], R = ret[i];
    const float m = mask[i] ? 1.f : 0.f;
    const float vc = fmaxf(fminf(v, vo + clip), vo - clip);
    const float l1 = (v - R) * (v - R), l2 = (vc - R) * (vc - R);
    const bool use2 = l2 > l1;
    float g = use2 ? ((vc == v) ? (v - R) : 0.f) : (v - R);
    grad_unnorm[i] = g * m;     // d(0.5 * l)/dv
    s[0] += fmaxf(l1, l2) * m; s[1] += m; s[2] += use2 ? m : 0.f;
  }
  double t[3];
  if (!loss_sums(s, scratch, t)) return;
  loss[0] = static_cast<float>(0.5 * t[0] / t[1]);
  stats[0] = static_cast<float>(t[1]);
  stats[1] = static_cast<float>(t[2] / t[1]);
}

// out = grad_unnorm * (g_loss / sum(m))
__global__ void loss_grad_kernel(const float* __restrict__ grad_unnorm, const float* __restrict__ g_loss, const float* __restrict__ denom,
                                 long n, float* __restrict__ out) {
  const float f = __fdiv_rn(g_loss[0], denom[0]);
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n; i += static_cast<long>(gridDim.x) * blockDim.x)
    out[i] = grad_unnorm[i] * f;
}

// blocks of a loss launch: one cluster (`scratch` unused) or many blocks
template <typename K, typename... Args>
cudaError_t launch_loss(K kern, long n, double* scratch, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kLossThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  unsigned blocks = 1;
  if (n <= kLossClusterMax) {
    while (blocks < 8 && static_cast<long>(blocks) * kLossThreads * 2 < n) blocks *= 2;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    scratch = nullptr;
  } else {
    blocks = kLossBlocks;
    cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
  }
  cfg.gridDim = dim3(blocks);
  return cudaLaunchKernelEx(&cfg, kern, args..., scratch);
}

// ---- AdamW over flat buffers --------------------------------------------------------------------
template <typename MomentT>
struct MomentIO;
template <>
struct MomentIO<float> {
  static NRL_DEVICE void load8(const float* p, float (&o)[8]) {
    float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
  }
  static NRL_DEVICE void store8(float* p, const float (&o)[8]) {
    reinterpret_cast<float4*>(p)[0] = make_float4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(o[4], o[5], o[6], o[7]);
  }
};
template <>
struct MomentIO<__nv_bfloat16> {
  static NRL_DEVICE void load8(const __nv_bfloat16* p, float (&o)[8]) {
    uint4 a = *reinterpret_cast<const uint4*>(p);
    uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = unpack_bf16x2(w[j]);
      o[2 * j] = f.x; o[2 * j + 1] = f.y;
    }
  }
  static NRL_DEVICE void store8(__nv_bfloat16* p, const float (&o)[8]) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]),
                                              pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
  }
};

NRL_DEVICE void adamw_update8(float (&p)[8], const float (&g)[8], float (&m)[8], float (&v)[8], const AdamHyper& h) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float gj = g[j] * h.grad_scale;
    m[j] = h.beta1 * m[j] + (1.f - h.beta1) * gj;
    v[j] = h.beta2 * v[j] + (1.f - h.beta2) * gj * gj;
    const float denom = sqrtf(v[j] * h.inv_bc2) + h.eps;
    p[j] = p[j] * (1.f - h.lr * h.wd) - h.step_size * (m[j] / denom);
  }
}

template <typename MomentT>
__global__ void adamw_flat_kernel(__nv_bfloat16* __restrict__ param, const __nv_bfloat16* __restrict__ grad,
                                  MomentT* __restrict__ m, MomentT* __restrict__ v, float* __restrict__ master, long n,
                                  AdamHyper h) {
  const long nvec = n / 8;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nvec;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    float p8[8], g8[8], m8[8], v8[8];
    if (master != nullptr) MomentIO<float>::load8(master + i * 8, p8);      // fp32 master weights (see comm.cu)
    else MomentIO<__nv_bfloat16>::load8(param + i * 8, p8);
    MomentIO<__nv_bfloat16>::load8(grad + i * 8, g8);
    MomentIO<MomentT>::load8(m + i * 8, m8);
    MomentIO<MomentT>::load8(v + i * 8, v8);
    adamw_update8(p8, g8, m8, v8, h);
    MomentIO<__nv_bfloat16>::store8(param + i * 8, p8);
    if (master != nullptr) MomentIO<float>::store8(master + i * 8, p8);
    MomentIO<MomentT>::store8(m + i * 8, m8);
    MomentIO<MomentT>::store8(v + i * 8, v8);
  }
}

}  // namespace nrl

using namespace nrl;

extern "C" cudaError_t nrl_gae_scan(const float* rewards, const float* values, float* adv, float* returns, int B,
                                    int T, double gamma, double lam, cudaStream_t s) {
  if (B == 0 || T == 0) return cudaSuccess;
  if (T <= 32 * kGaePer)
    gae_scan_kernel<1><<<(B + kGaeRows - 1) / kGaeRows, 32 * kGaeRows, 0, s>>>(rewards, values, adv, returns, B, T, gamma, lam);
  else
    gae_scan_kernel<kGaeWarps><<<B, 32 * kGaeWarps, 0, s>>>(rewards, values, adv, returns, B, T, gamma, lam);
  return cudaGetLastError();
}

extern "C" long nrl_loss_scratch_doubles(long n) { return n <= kLossClusterMax ? 0 : 1 + 9L * kLossBlocks; }

extern "C" cudaError_t nrl_policy_loss(const float* new_lp, const float* old_lp, const float* adv,
                                       const uint8_t* mask, const float* ref_lp, float cliprange, float kl_coef,
                                       long n, float* grad_unnorm, float* loss, float* stats, double* scratch, cudaStream_t s) {
  return launch_loss(policy_loss_kernel, n, scratch, s, new_lp, old_lp, adv, mask, ref_lp, cliprange, kl_coef, n, grad_unnorm, loss, stats);
}

extern "C" cudaError_t nrl_value_loss(const float* vpred, const float* vold, const float* ret, const uint8_t* mask,
                                      float clip, long n, float* grad_unnorm, float* loss, float* stats, double* scratch, cudaStream_t s) {
  return launch_loss(value_loss_kernel, n, scratch, s, vpred, vold, ret, mask, clip, n, grad_unnorm, loss, stats);
}

extern "C" cudaError_t nrl_loss_grad(const float* grad_unnorm, const float* g_loss, const float* denom, long n, float* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  long blocks = (n + 255) / 256;
  if (blocks > 296) blocks = 296;
  loss_grad_kernel<<<static_cast<int>(blocks), 256, 0, s>>>(grad_unnorm, g_loss, denom, n, out);
  return cudaGetLastError();
}

extern "C" cudaError_t nrl_adamw_flat(void* param, const void* grad, void* m, void* v, float* master, long n,
                                      int moments_bf16, AdamHyper h, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (n % 8 != 0) return cudaErrorInvalidValue;
  long blocks = (n / 8 + 255) / 256;
  if (blocks > 148L * 8) blocks = 148L * 8;
  auto P = static_cast<__nv_bfloat16*>(param);
  auto G = static_cast<const __nv_bfloat16*>(grad);
  if (moments_bf16)
    adamw_flat_kernel<__nv_bfloat16><<<static_cast<int>(blocks), 256, 0, s>>>(
        P, G, static_cast<__nv_bfloat16*>(m), static_cast<__nv_bfloat16*>(v), master, n, h);
  else
    adamw_flat_kernel<float><<<static_cast<int>(blocks), 256, 0, s>>>(P, G, static_cast<float*>(m),
                                                                       static_cast<float*>(v), master, n, h);
  return cudaGetLastError();
}
