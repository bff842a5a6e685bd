// Recurrent token mixers with state carried per sequence slot: short causal convolution, state-space scan with a scalar
// decay per head, gated delta rule with a decay per head or per key channel.  One launch serves a whole engine step:
// every entry (a run of consecutive tokens of one sequence: a prompt portion or one decoded token) starts from the state
// its slot holds (zero when the sequence is new) and leaves the updated state there.  All arithmetic is float.
// Compiled WITHOUT fast-math.
#include <cuda_bf16.h>

#include "hybrid_kernels.h"

namespace {

constexpr int kMaxTaps = 16;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ---------------------------------------------------------------------------------------------------------------------
// causal convolution: thread per (token, channel)
// ---------------------------------------------------------------------------------------------------------------------
__global__ void causal_conv_kernel(const float* __restrict__ in, long si, const float* __restrict__ in_bias, int act,
                                   const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ state, float* __restrict__ out, long so, const int* __restrict__ cu,
                                   const int* __restrict__ tok_entry, const int* __restrict__ start,
                                   const int* __restrict__ state_slot, long T, int C, int taps) {
  const long idx = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (idx >= T * C) return;
  const long t = idx / C;
  const int c = static_cast<int>(idx - t * C);
  const int e = tok_entry[t];
  const long first = cu[e];
  const int local = static_cast<int>(t - first);
  const bool carried = start[e] > 0;
  const float* st = state + static_cast<long>(state_slot[e]) * (taps - 1) * C;
  float acc = bias != nullptr ? bias[c] : 0.f;
  const float ib = in_bias != nullptr ? in_bias[c] : 0.f;
  for (int j = 0; j < taps; ++j) {
    const int src = local - (taps - 1 - j);
    float x = 0.f;
    if (src >= 0) x = in[(first + src) * si + c] + ib;
    else if (carried) x = st[static_cast<long>(taps - 1 + src) * C + c];
    acc += w[static_cast<long>(c) * taps + j] * x;
  }
  out[t * so + c] = act ? silu(acc) : acc;
}

// thread per (channel, run of kConvTok consecutive tokens): the last taps-1 inputs slide through registers, so every input is
// read once (plus the history at the start of a run or of a sequence) and the taps' weights once per run
constexpr int kConvTok = 8;

template <int MAXT>
__global__ void causal_conv_run_kernel(const float* __restrict__ in, long si, const float* __restrict__ in_bias, int act,
                                       const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ state, float* __restrict__ out, long so, const int* __restrict__ cu,
                                       const int* __restrict__ tok_entry, const int* __restrict__ start,
                                       const int* __restrict__ state_slot, int T, int C, int taps) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int t_begin = blockIdx.y * kConvTok, t_end = min(T, t_begin + kConvTok);
  float wv[MAXT], hist[MAXT];
#pragma unroll
  for (int j = 0; j < MAXT; ++j) {
    wv[j] = j < taps ? w[static_cast<long>(c) * taps + j] : 0.f;
    hist[j] = 0.f;
  }
  const float b = bias != nullptr ? bias[c] : 0.f;
  const float ib = in_bias != nullptr ? in_bias[c] : 0.f;
  int e_prev = -1;
  for (int t = t_begin; t < t_end; ++t) {
    const int e = tok_entry[t];
    if (e != e_prev) {                                   // first token of the run, or another sequence begins: fetch the history
      const long first = cu[e];
      const int local = static_cast<int>(t - first);
      const bool carried = start[e] > 0;
      const float* st = state + static_cast<long>(state_slot[e]) * (taps - 1) * C;
#pragma unroll
      for (int j = 0; j < MAXT - 1; ++j) {
        if (j < taps - 1) {
          const int src = local - (taps - 1 - j);
          float x = 0.f;
          if (src >= 0) x = in[(first + src) * si + c] + ib;
          else if (carried) x = st[static_cast<long>(taps - 1 + src) * C + c];
          hist[j] = x;
        }
      }
      e_prev = e;
    }
    const float cur = in[static_cast<long>(t) * si + c] + ib;
    float acc = b;
#pragma unroll
    for (int j = 0; j < MAXT - 1; ++j)
      if (j < taps - 1) acc += wv[j] * hist[j];
#pragma unroll
    for (int j = 0; j < MAXT; ++j)
      if (j == taps - 1) acc += wv[j] * cur;
    out[static_cast<long>(t) * so + c] = act ? silu(acc) : acc;
#pragma unroll
    for (int j = 0; j < MAXT - 1; ++j) {
      if (j < taps - 2) hist[j] = hist[j + 1];
      else if (j == taps - 2) hist[j] = cur;
    }
  }
}

// thread per (entry, channel): the slot keeps the last taps-1 inputs of the sequence, oldest first
__global__ void causal_conv_carry_kernel(const float* __restrict__ in, long si, const float* __restrict__ in_bias,
                                         float* __restrict__ state, const int* __restrict__ cu,
                                         const int* __restrict__ start, const int* __restrict__ state_slot, int E, int C, int taps) {
  const long idx = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (idx >= static_cast<long>(E) * C) return;
  const int e = static_cast<int>(idx / C);
  const int c = static_cast<int>(idx - static_cast<long>(e) * C);
  const long first = cu[e];
  const int n = cu[e + 1] - cu[e];
  const bool carried = start[e] > 0;
  float* st = state + static_cast<long>(state_slot[e]) * (taps - 1) * C;
  float keep[kMaxTaps];
  const float ib = in_bias != nullptr ? in_bias[c] : 0.f;
#pragma unroll
  for (int j = 0; j < kMaxTaps; ++j) {
    if (j < taps - 1) {
      const int src = n - (taps - 1) + j;
      float x = 0.f;
      if (src >= 0) x = in[(first + src) * si + c] + ib;
      else if (carried) x = st[static_cast<long>(taps - 1 + src) * C + c];
      keep[j] = x;
    }
  }
#pragma unroll
  for (int j = 0; j < kMaxTaps; ++j)
    if (j < taps - 1) st[static_cast<long>(j) * C + c] = keep[j];
}

// ---------------------------------------------------------------------------------------------------------------------
// state-space scan: block per (entry, head); thread (r, p) owns column p of S [N, P] for rows n = r, r + R, ...
// ---------------------------------------------------------------------------------------------------------------------
__global__ void ssd_scan_kernel(const float* __restrict__ xbc, long sx, int col_b, int col_c, const float* __restrict__ dt_raw, long sd,
                                const float* __restrict__ dt_bias, const float* __restrict__ A_log, const float* __restrict__ Dskip,
                                float* __restrict__ state, float* __restrict__ y, const int* __restrict__ cu,
                                const int* __restrict__ start, const int* __restrict__ state_slot, int heads, int groups, int N, int P,
                                int R) {
  extern __shared__ float sm[];
  float* S = sm;                         // [N][P]
  float* vB = S + static_cast<long>(N) * P;   // [N]
  float* vC = vB + N;                    // [N]
  float* vx = vC + N;                    // [P]
  float* red = vx + P;                   // [R][P]
  const int e = blockIdx.x, h = blockIdx.y, g = h / (heads / groups);
  const int tid = threadIdx.x, r = tid / P, p = tid - r * P;
  const bool live = r < R;
  float* gS = state + (static_cast<long>(state_slot[e]) * heads + h) * N * P;
  const bool carried = start[e] > 0;
  for (int i = tid; i < N * P; i += blockDim.x) S[i] = carried ? gS[i] : 0.f;
  const float negA = -expf(A_log[h]), dskip = Dskip[h], bias = dt_bias[h];
  const int t0 = cu[e], t1 = cu[e + 1];
  for (int t = t0; t < t1; ++t) {
    __syncthreads();                                                     // S loaded / previous token's reads done
    const float* row = xbc + static_cast<long>(t) * sx;
    for (int i = tid; i < N; i += blockDim.x) {
      vB[i] = row[col_b + g * N + i];
      vC[i] = row[col_c + g * N + i];
    }
    for (int i = tid; i < P; i += blockDim.x) vx[i] = row[h * P + i];
    const float dt = softplus(dt_raw[static_cast<long>(t) * sd + h] + bias);
    const float a = expf(negA * dt);
    __syncthreads();
    float acc = 0.f;
    if (live) {
      const float xs = dt * vx[p];
      for (int n = r; n < N; n += R) {
        const float sv = a * S[n * P + p] + vB[n] * xs;
        S[n * P + p] = sv;
        acc += sv * vC[n];
      }
      red[r * P + p] = acc;
    }
    __syncthreads();
    if (tid < P) {
      float tot = 0.f;
      for (int q = 0; q < R; ++q) tot += red[q * P + tid];
      y[static_cast<long>(t) * heads * P + h * P + tid] = tot + dskip * vx[tid];
    }
  }
  __syncthreads();
  for (int i = tid; i < N * P; i += blockDim.x) gS[i] = S[i];
}

// ---------------------------------------------------------------------------------------------------------------------
// gated delta rule
// ---------------------------------------------------------------------------------------------------------------------
// block per token: warps normalise the q / k heads, then all threads form beta and the decays
__global__ void delta_prep_kernel(float* __restrict__ qkv, long sq, int col_k, const float* __restrict__ b_raw, long sb,
                                  const float* __restrict__ a_raw, long sa, const float* __restrict__ dt_bias,
                                  const float* __restrict__ A_log, float* __restrict__ beta, float* __restrict__ decay, int heads,
                                  int kv_heads, int D, int per_channel) {
  const long t = blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float qscale = 1.f / sqrtf(static_cast<float>(D));
  for (int hh = w; hh < 2 * kv_heads; hh += nw) {
    const bool is_k = hh >= kv_heads;
    float* v = qkv + t * sq + (is_k ? col_k + (hh - kv_heads) * D : hh * D);
    float ss = 0.f;
    for (int c = lane; c < D; c += 32) ss += v[c] * v[c];
    ss = warp_sum(ss);
    const float r = (is_k ? 1.f : qscale) / sqrtf(ss + 1e-6f);
    for (int c = lane; c < D; c += 32) v[c] *= r;
  }
  for (int hh = threadIdx.x; hh < heads; hh += blockDim.x) beta[t * heads + hh] = 1.f / (1.f + expf(-b_raw[t * sb + hh]));
  const int nd = per_channel ? heads * D : heads;
  for (int i = threadIdx.x; i < nd; i += blockDim.x) {
    const int hh = per_channel ? i / D : i;
    decay[t * nd + i] = expf(-expf(A_log[hh]) * softplus(a_raw[t * sa + i] + dt_bias[i]));
  }
}

// Gated linear attention inputs, block per token: q (columns 0 .. heads*D-1 of qkv, in place) times D^-1/2, and the decay of every
// key channel  decay[t, i] = sigmoid(z)^(1 / tau) = exp(-softplus(-z) / tau)  with z = a_raw[t, i] + a_bias[i].
__global__ void gla_prep_kernel(float* __restrict__ qkv, long sq, const float* __restrict__ a_raw, long sa, const float* __restrict__ a_bias,
                                float inv_tau, float* __restrict__ decay, int n, int D) {
  const long t = blockIdx.x;
  const float qscale = 1.f / sqrtf(static_cast<float>(D));
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    qkv[t * sq + i] *= qscale;
    const float z = a_raw[t * sa + i] + (a_bias != nullptr ? a_bias[i] : 0.f);
    decay[t * n + i] = expf(-softplus(-z) * inv_tau);
  }
}

// block per (entry, head); thread (r, v) owns column v of S [D, Dv] for rows d = r, r + R, ...
// One pass over S forms the decayed state, S^T k and S^T q; the read-out of the written state is o = S^T q + u (k . q).
__global__ void delta_scan_kernel(const float* __restrict__ qkv, long sq, int col_k, int col_v, const float* __restrict__ beta,
                                  const float* __restrict__ decay, float* __restrict__ state, float* __restrict__ o,
                                  const int* __restrict__ cu, const int* __restrict__ start, const int* __restrict__ state_slot,
                                  int heads, int kv_heads, int D, int Dv, int per_channel, int R) {
  extern __shared__ float sm[];
  float* S = sm;                              // [D][Dv]
  float* vq = S + static_cast<long>(D) * Dv;  // [D]
  float* vk = vq + D;                         // [D]
  float* vg = vk + D;                         // [D]
  float* red = vg + D;                        // [2][R][Dv]
  float* kq = red + 2 * R * Dv;               // [1]
  const int e = blockIdx.x, h = blockIdx.y, g = h / (heads / kv_heads);
  const int tid = threadIdx.x, r = tid / Dv, v = tid - r * Dv;
  const bool live = r < R;
  float* gS = state + (static_cast<long>(state_slot[e]) * heads + h) * D * Dv;
  const bool carried = start[e] > 0;
  for (int i = tid; i < D * Dv; i += blockDim.x) S[i] = carried ? gS[i] : 0.f;
  const int t0 = cu[e], t1 = cu[e + 1];
  const int nd = per_channel ? heads * D : heads;
  for (int t = t0; t < t1; ++t) {
    __syncthreads();
    const float* row = qkv + static_cast<long>(t) * sq;
    for (int i = tid; i < D; i += blockDim.x) {
      vq[i] = row[g * D + i];
      vk[i] = row[col_k + g * D + i];
      vg[i] = per_channel ? decay[static_cast<long>(t) * nd + h * D + i] : decay[static_cast<long>(t) * nd + h];
    }
    __syncthreads();
    if (tid < 32) {
      float d = 0.f;
      for (int i = tid; i < D; i += 32) d += vk[i] * vq[i];
      d = warp_sum(d);
      if (tid == 0) kq[0] = d;
    }
    float pk = 0.f, pq = 0.f;
    if (live) {
      for (int d = r; d < D; d += R) {
        const float sv = vg[d] * S[d * Dv + v];
        S[d * Dv + v] = sv;
        pk += sv * vk[d];
        pq += sv * vq[d];
      }
      red[r * Dv + v] = pk;
      red[(R + r) * Dv + v] = pq;
    }
    __syncthreads();
    if (live) {
      float sk = 0.f, sq_ = 0.f;
      for (int q = 0; q < R; ++q) {
        sk += red[q * Dv + v];
        sq_ += red[(R + q) * Dv + v];
      }
      const float vt = row[col_v + h * Dv + v];
      const float u = beta != nullptr ? beta[static_cast<long>(t) * heads + h] * (vt - sk) : vt;   // no beta: plain accumulation
      if (r == 0) o[static_cast<long>(t) * heads * Dv + h * Dv + v] = sq_ + u * kq[0];
      for (int d = r; d < D; d += R) S[d * Dv + v] += vk[d] * u;
    }
  }
  __syncthreads();
  for (int i = tid; i < D * Dv; i += blockDim.x) gS[i] = S[i];
}


// ---------------------------------------------------------------------------------------------------------------------
// Register-resident scans (the usual sizes): thread (r, c) keeps rows r, r + R, ... of column c of the state in RPT
// registers for the whole entry -- one global read of the state at the start, one write at the end, which is all a decoded
// token needs -- and the next token's inputs are fetched into registers while the current token is computed.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kPre = 4;            // prefetch registers per thread

template <int RPT>
__global__ void __launch_bounds__(RPT >= 64 ? 256 : 512)
ssd_scan_reg_kernel(const float* __restrict__ xbc, long sx, int col_b, int col_c, const float* __restrict__ dt_raw, long sd,
                    const float* __restrict__ dt_bias, const float* __restrict__ A_log, const float* __restrict__ Dskip,
                    float* __restrict__ state, float* __restrict__ y, const int* __restrict__ cu, const int* __restrict__ start,
                    const int* __restrict__ state_slot, int heads, int groups, int N, int P, int R) {
  extern __shared__ float sm[];
  const int L = 2 * N + P;                       // per token: B | C | x
  float* vec = sm;                               // [2][L]
  float* red = sm + 2 * L;                       // [R][P]
  const int e = blockIdx.x, h = blockIdx.y, g = h / (heads / groups);
  const int tid = threadIdx.x, nth = blockDim.x, r = tid / P, p = tid - r * P;
  const bool live = r < R;
  float* gS = state + (static_cast<long>(state_slot[e]) * heads + h) * N * P;
  const bool carried = start[e] > 0;
  float S[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int n = r + i * R;
    S[i] = (live && n < N && carried) ? gS[n * P + p] : 0.f;
  }
  const float negA = -expf(A_log[h]), dskip = Dskip[h], bias = dt_bias[h];
  const int t0 = cu[e], t1 = cu[e + 1];
  auto src = [&](int t, int idx) -> const float* {
    const float* row = xbc + static_cast<long>(t) * sx;
    return idx < N ? row + col_b + g * N + idx : idx < 2 * N ? row + col_c + g * N + (idx - N) : row + h * P + (idx - 2 * N);
  };
  float pre[kPre], pre_dt;
#pragma unroll
  for (int i = 0; i < kPre; ++i) {
    const int idx = tid + i * nth;
    pre[i] = idx < L ? *src(t0, idx) : 0.f;
  }
  pre_dt = dt_raw[static_cast<long>(t0) * sd + h];
  for (int t = t0; t < t1; ++t) {
    float* v = vec + ((t - t0) & 1) * L;
#pragma unroll
    for (int i = 0; i < kPre; ++i) {
      const int idx = tid + i * nth;
      if (idx < L) v[idx] = pre[i];
    }
    const float dt = softplus(pre_dt + bias);
    __syncthreads();
    if (t + 1 < t1) {
#pragma unroll
      for (int i = 0; i < kPre; ++i) {
        const int idx = tid + i * nth;
        if (idx < L) pre[i] = *src(t + 1, idx);
      }
      pre_dt = dt_raw[static_cast<long>(t + 1) * sd + h];
    }
    const float a = expf(negA * dt);
    const float* vB = v;
    const float* vC = v + N;
    const float* vx = v + 2 * N;
    if (live) {
      const float xs = dt * vx[p];
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int n = r + i * R;
        if (n < N) {
          S[i] = a * S[i] + vB[n] * xs;
          acc += S[i] * vC[n];
        }
      }
      red[r * P + p] = acc;
    }
    __syncthreads();
    if (tid < P) {
      float tot = 0.f;
      for (int q = 0; q < R; ++q) tot += red[q * P + tid];
      y[static_cast<long>(t) * heads * P + h * P + tid] = tot + dskip * vx[tid];
    }
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int n = r + i * R;
      if (n < N) gS[n * P + p] = S[i];
    }
  }
}

template <int RPT>
__global__ void __launch_bounds__(RPT >= 64 ? 256 : 512)
delta_scan_reg_kernel(const float* __restrict__ qkv, long sq, int col_k, int col_v, const float* __restrict__ beta,
                      const float* __restrict__ decay, float* __restrict__ state, float* __restrict__ o, const int* __restrict__ cu,
                      const int* __restrict__ start, const int* __restrict__ state_slot, int heads, int kv_heads, int D, int Dv,
                      int per_channel, int R) {
  extern __shared__ float sm[];
  const int L = 3 * D;                           // per token: q | k | decay per row
  float* vec = sm;                               // [2][L]
  float* red = sm + 2 * L;                       // [2][R][Dv]
  float* rkq = red + 2 * R * Dv;                 // [R]
  const int e = blockIdx.x, h = blockIdx.y, g = h / (heads / kv_heads);
  const int tid = threadIdx.x, nth = blockDim.x, r = tid / Dv, c = tid - r * Dv;
  const bool live = r < R;
  float* gS = state + (static_cast<long>(state_slot[e]) * heads + h) * D * Dv;
  const bool carried = start[e] > 0;
  float S[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int d = r + i * R;
    S[i] = (live && d < D && carried) ? gS[d * Dv + c] : 0.f;
  }
  const int t0 = cu[e], t1 = cu[e + 1];
  const int nd = per_channel ? heads * D : heads;
  auto src = [&](int t, int idx) -> const float* {
    const float* row = qkv + static_cast<long>(t) * sq;
    return idx < D ? row + g * D + idx
           : idx < 2 * D ? row + col_k + g * D + (idx - D)
                         : decay + static_cast<long>(t) * nd + (per_channel ? h * D + (idx - 2 * D) : h);
  };
  float pre[kPre], pre_v = 0.f, pre_beta;
#pragma unroll
  for (int i = 0; i < kPre; ++i) {
    const int idx = tid + i * nth;
    pre[i] = idx < L ? *src(t0, idx) : 0.f;
  }
  if (live) pre_v = qkv[static_cast<long>(t0) * sq + col_v + h * Dv + c];
  pre_beta = beta != nullptr ? beta[static_cast<long>(t0) * heads + h] : 0.f;
  for (int t = t0; t < t1; ++t) {
    float* v = vec + ((t - t0) & 1) * L;
#pragma unroll
    for (int i = 0; i < kPre; ++i) {
      const int idx = tid + i * nth;
      if (idx < L) v[idx] = pre[i];
    }
    const float v_cur = pre_v, b_cur = pre_beta;
    __syncthreads();
    if (t + 1 < t1) {
#pragma unroll
      for (int i = 0; i < kPre; ++i) {
        const int idx = tid + i * nth;
        if (idx < L) pre[i] = *src(t + 1, idx);
      }
      if (live) pre_v = qkv[static_cast<long>(t + 1) * sq + col_v + h * Dv + c];
      pre_beta = beta != nullptr ? beta[static_cast<long>(t + 1) * heads + h] : 0.f;
    }
    const float* vq = v;
    const float* vk = v + D;
    const float* vg = v + 2 * D;
    if (live) {
      float pk = 0.f, pq = 0.f, pkq = 0.f;
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int d = r + i * R;
        if (d < D) {
          const float sv = vg[d] * S[i];
          S[i] = sv;
          pk += sv * vk[d];
          pq += sv * vq[d];
          if (c == 0) pkq += vk[d] * vq[d];
        }
      }
      red[r * Dv + c] = pk;
      red[(R + r) * Dv + c] = pq;
      if (c == 0) rkq[r] = pkq;
    }
    __syncthreads();
    if (live) {
      float sk = 0.f, sq_ = 0.f, kq = 0.f;
      for (int x = 0; x < R; ++x) {
        sk += red[x * Dv + c];
        sq_ += red[(R + x) * Dv + c];
        kq += rkq[x];
      }
      const float u = beta != nullptr ? b_cur * (v_cur - sk) : v_cur;
      if (r == 0) o[static_cast<long>(t) * heads * Dv + h * Dv + c] = sq_ + u * kq;
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int d = r + i * R;
        if (d < D) S[i] += vk[d] * u;
      }
    }
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int d = r + i * R;
      if (d < D) gS[d * Dv + c] = S[i];
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Column-resident scans (state rows <= 128, the usual sizes): thread c keeps the whole column c of the state in ROWS
// registers, so S^T k, S^T q and S^T C are sums inside one thread -- no reduction across threads -- and a token costs one
// barrier: the vectors all columns share (B and C, or q, k and the row decays) are staged in shared memory, double
// buffered, zero padded to ROWS, and fetched from global memory one token ahead.
// ---------------------------------------------------------------------------------------------------------------------
__host__ __device__ constexpr int col_min_threads(int rows) { return rows > 64 ? 64 : 32; }      // so that a thread stages few values per token

// SPLIT (1 or 2) threads share a column: neighbouring lanes hold the upper and the lower half of its rows and add their
// partial sums with one shuffle (more threads in flight and half the registers for 128-row states).  In shared memory a
// staged vector is SPLIT segments of ROWS / SPLIT + 4 floats, so that the two halves read different banks.
template <int ROWS, int SPLIT>
struct ColStage {
  static constexpr int RH = ROWS / SPLIT;                 // rows per thread
  static constexpr int VL = SPLIT * (RH + 4);             // floats per staged vector
  __host__ __device__ static constexpr int at(int d) { return (d / RH) * (RH + 4) + d % RH; }
};

template <int ROWS, int SPLIT>
__global__ void __launch_bounds__(256)
ssd_scan_col_kernel(const float* __restrict__ xbc, long sx, int col_b, int col_c, const float* __restrict__ dt_raw, long sd,
                    const float* __restrict__ dt_bias, const float* __restrict__ A_log, const float* __restrict__ Dskip,
                    float* __restrict__ state, float* __restrict__ y, const int* __restrict__ cu, const int* __restrict__ start,
                    const int* __restrict__ state_slot, int heads, int groups, int N, int P) {
  using St = ColStage<ROWS, SPLIT>;
  constexpr int RH = St::RH, VL = St::VL, L = 2 * VL + 4;  // per token: B | C | dt, decay
  constexpr int kStagePre = (2 * ROWS + col_min_threads(ROWS) - 1) / col_min_threads(ROWS);
  __shared__ __align__(16) float stage[2 * L];
  const int e = blockIdx.x, h = blockIdx.y, g = h / (heads / groups);
  const int tid = threadIdx.x, nth = blockDim.x, p = tid / SPLIT, half = tid % SPLIT, r0 = half * RH;
  const bool live = p < P;
  float* gS = state + (static_cast<long>(state_slot[e]) * heads + h) * N * P;
  const bool carried = start[e] > 0;
  float S[RH];
#pragma unroll
  for (int i = 0; i < RH; ++i) S[i] = (live && r0 + i < N && carried) ? gS[static_cast<long>(r0 + i) * P + p] : 0.f;
  const float negA = -expf(A_log[h]), dskip = Dskip[h], bias = dt_bias[h];
  const int t0 = cu[e], t1 = cu[e + 1];
  float pre[kStagePre], pre_x, pre_dt;
  auto fetch = [&](int t) {
    const float* row = xbc + static_cast<long>(t) * sx;
#pragma unroll
    for (int i = 0; i < kStagePre; ++i) {
      const int idx = tid + i * nth;
      if (idx < 2 * ROWS) {
        const int n = idx < ROWS ? idx : idx - ROWS;
        pre[i] = n < N ? row[(idx < ROWS ? col_b : col_c) + g * N + n] : 0.f;
      }
    }
    pre_x = live ? row[h * P + p] : 0.f;
    pre_dt = dt_raw[static_cast<long>(t) * sd + h];
  };
  if (t0 < t1) fetch(t0);
  for (int t = t0; t < t1; ++t) {
    float* v = stage + ((t - t0) & 1) * L;
#pragma unroll
    for (int i = 0; i < kStagePre; ++i) {
      const int idx = tid + i * nth;
      if (idx < 2 * ROWS) v[(idx < ROWS ? 0 : VL) + St::at(idx < ROWS ? idx : idx - ROWS)] = pre[i];
    }
    if (tid == 0) {
      const float dt = softplus(pre_dt + bias);
      v[2 * VL] = dt;
      v[2 * VL + 1] = expf(negA * dt);
    }
    const float x_cur = pre_x;
    __syncthreads();
    if (t + 1 < t1) fetch(t + 1);
    const float dt = v[2 * VL], a = v[2 * VL + 1];
    const float xs = dt * x_cur;
    const float4* vB = reinterpret_cast<const float4*>(v + half * (RH + 4));
    const float4* vC = reinterpret_cast<const float4*>(v + VL + half * (RH + 4));
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < RH / 4; ++i) {
      const float4 b = vB[i], c = vC[i];
      S[4 * i] = a * S[4 * i] + b.x * xs;
      S[4 * i + 1] = a * S[4 * i + 1] + b.y * xs;
      S[4 * i + 2] = a * S[4 * i + 2] + b.z * xs;
      S[4 * i + 3] = a * S[4 * i + 3] + b.w * xs;
      acc[0] += S[4 * i] * c.x;
      acc[1] += S[4 * i + 1] * c.y;
      acc[2] += S[4 * i + 2] * c.z;
      acc[3] += S[4 * i + 3] * c.w;
    }
    float tot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    if (SPLIT == 2) tot += __shfl_xor_sync(0xffffffffu, tot, 1);
    if (live && half == 0) y[static_cast<long>(t) * heads * P + h * P + p] = tot + dskip * x_cur;
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RH; ++i)
      if (r0 + i < N) gS[static_cast<long>(r0 + i) * P + p] = S[i];
  }
}

template <int ROWS, int SPLIT>
__global__ void __launch_bounds__(256)
delta_scan_col_kernel(const float* __restrict__ qkv, long sq, int col_k, int col_v, const float* __restrict__ beta,
                      const float* __restrict__ decay, float* __restrict__ state, float* __restrict__ o, const int* __restrict__ cu,
                      const int* __restrict__ start, const int* __restrict__ state_slot, int heads, int kv_heads, int D, int Dv,
                      int per_channel) {
  using St = ColStage<ROWS, SPLIT>;
  constexpr int RH = St::RH, VL = St::VL, L = 3 * VL;      // per token: q | k | row decays
  constexpr int kStagePre = (3 * ROWS + col_min_threads(ROWS) - 1) / col_min_threads(ROWS);
  __shared__ __align__(16) float stage[2 * L];
  const int e = blockIdx.x, h = blockIdx.y, g = h / (heads / kv_heads);
  const int tid = threadIdx.x, nth = blockDim.x, c = tid / SPLIT, half = tid % SPLIT, r0 = half * RH;
  const bool live = c < Dv;
  float* gS = state + (static_cast<long>(state_slot[e]) * heads + h) * D * Dv;
  const bool carried = start[e] > 0;
  float S[RH];
#pragma unroll
  for (int i = 0; i < RH; ++i) S[i] = (live && r0 + i < D && carried) ? gS[static_cast<long>(r0 + i) * Dv + c] : 0.f;
  const int t0 = cu[e], t1 = cu[e + 1];
  const int nd = per_channel ? heads * D : heads;
  float pre[kStagePre], pre_v, pre_beta;
  auto fetch = [&](int t) {
    const float* row = qkv + static_cast<long>(t) * sq;
#pragma unroll
    for (int i = 0; i < kStagePre; ++i) {
      const int idx = tid + i * nth;
      if (idx < 3 * ROWS) {
        const int part = idx / ROWS, d = idx - part * ROWS;
        float x = 0.f;
        if (d < D) {
          if (part == 0) x = row[g * D + d];
          else if (part == 1) x = row[col_k + g * D + d];
          else x = decay[static_cast<long>(t) * nd + (per_channel ? h * D + d : h)];
        }
        pre[i] = x;
      }
    }
    pre_v = live ? row[col_v + h * Dv + c] : 0.f;
    pre_beta = beta != nullptr ? beta[static_cast<long>(t) * heads + h] : 0.f;
  };
  if (t0 < t1) fetch(t0);
  for (int t = t0; t < t1; ++t) {
    float* v = stage + ((t - t0) & 1) * L;
#pragma unroll
    for (int i = 0; i < kStagePre; ++i) {
      const int idx = tid + i * nth;
      if (idx < 3 * ROWS) v[(idx / ROWS) * VL + St::at(idx % ROWS)] = pre[i];
    }
    const float v_cur = pre_v, b_cur = pre_beta;
    __syncthreads();
    if (t + 1 < t1) fetch(t + 1);
    const float4* vq = reinterpret_cast<const float4*>(v + half * (RH + 4));
    const float4* vk = reinterpret_cast<const float4*>(v + VL + half * (RH + 4));
    const float4* vg = reinterpret_cast<const float4*>(v + 2 * VL + half * (RH + 4));
    float pk[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < RH / 4; ++i) {                         // S <- g S;  S^T k
      const float4 gg = vg[i], kk = vk[i];
      S[4 * i] *= gg.x;
      S[4 * i + 1] *= gg.y;
      S[4 * i + 2] *= gg.z;
      S[4 * i + 3] *= gg.w;
      pk[0] += S[4 * i] * kk.x;
      pk[1] += S[4 * i + 1] * kk.y;
      pk[2] += S[4 * i + 2] * kk.z;
      pk[3] += S[4 * i + 3] * kk.w;
    }
    float sk = (pk[0] + pk[1]) + (pk[2] + pk[3]);
    if (SPLIT == 2) sk += __shfl_xor_sync(0xffffffffu, sk, 1);
    const float u = beta != nullptr ? b_cur * (v_cur - sk) : v_cur;
    float po[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < RH / 4; ++i) {                         // S <- S + k u^T;  o = S^T q sees this token's write
      const float4 kk = vk[i], qq = vq[i];
      S[4 * i] += kk.x * u;
      S[4 * i + 1] += kk.y * u;
      S[4 * i + 2] += kk.z * u;
      S[4 * i + 3] += kk.w * u;
      po[0] += S[4 * i] * qq.x;
      po[1] += S[4 * i + 1] * qq.y;
      po[2] += S[4 * i + 2] * qq.z;
      po[3] += S[4 * i + 3] * qq.w;
    }
    float so_ = (po[0] + po[1]) + (po[2] + po[3]);
    if (SPLIT == 2) so_ += __shfl_xor_sync(0xffffffffu, so_, 1);
    if (live && half == 0) o[static_cast<long>(t) * heads * Dv + h * Dv + c] = so_;
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RH; ++i)
      if (r0 + i < D) gS[static_cast<long>(r0 + i) * Dv + c] = S[i];
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Delta rule (or plain accumulation) of prompt portions, four tokens at a time, all arithmetic float.  With g_i the decays, c_i = g_1 .. g_i
// and G(i, j) = g_{j+1} .. g_i (products, nothing is divided), tokens 1..4 of a chunk over the state S before it give
//   u_i = beta_i (v_i - S^T (c_i k_i) - sum_{j<i} (k_i . G(i,j) k_j) u_j)          (no delta: u_i = v_i)
//   o_i = S^T (c_i q_i) + sum_{j<=i} (q_i . G(i,j) k_j) u_j
//   S  <- c_4 S + sum_j (G(4,j) k_j) u_j^T
// so an element of the state costs three multiply-adds per token (and one product per chunk) and every vector value that is read from
// shared memory serves four or eight columns.  The column-resident kernels wait for their vectors and two sums once per token: 16 x 2048
// tokens, 16 heads of 128 x 128: 4350 us there, 2300 us here (950 us at the float32 multiply-add rate).  What bounds it now is latency and
// registers: 128 rows x 8 columns take 254 and spill (-Xptxas -v: 870 to 950 bytes of stores and 1200 to 1350 of loads a thread; 4 columns of 128 rows and 8 of
// 64 about 300 to 400 each), so eight warps per SM issue 0.38 instructions per clock and scheduler, stalled on shared-memory reads, shuffles and fixed latencies.
// Inputs come by cp.async three chunks ahead and a chunk's vectors are prepared while the one before is computed (2520 us with loads one
// chunk ahead); 64 registers of state per thread over twice the warps took 2730 us.
//
// Lane = (one of four column groups, one of eight row groups): a thread keeps 2 PIECES rows x CT columns of the state in registers, rows
// 16 p + 2 rg + {0, 1}, columns in pairs for the packed multiply-add; the shared vectors are stored with every value twice, so that
// a 16-byte read is two ready operands and serves 2 x CT columns.  Sums over the row groups go by reduce-scatter shuffles: register a of a
// thread is column a ^ x of its group (x: the column the lane will own), which makes "the half to send" the same registers in every lane.
// Columns are independent: a state's columns are cut over blocks of two warps, 8 CT columns each.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kBlkTok = 4;
constexpr int kBlkWarps = 2;

__device__ __forceinline__ void cp_async_f32(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_f32x4(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// r[i] = sum over all rows of S[., column x] * v_i: `vec` holds four padded vectors with every value twice
template <int PIECES, int CT>
__device__ __forceinline__ void blk_product(const f32x2 (&S)[2 * PIECES][CT / 2], const float2* vec, int rg, float (&r)[kBlkTok]) {
  constexpr int DP = 16 * PIECES;
  f32x2 acc[CT / 2][kBlkTok];
#pragma unroll
  for (int a = 0; a < CT / 2; ++a)
#pragma unroll
    for (int i = 0; i < kBlkTok; ++i) acc[a][i] = 0;
#pragma unroll
  for (int pc = 0; pc < PIECES; ++pc)
#pragma unroll
    for (int i = 0; i < kBlkTok; ++i) {
      const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(vec + i * DP + pc * 16 + rg * 2);
#pragma unroll
      for (int a = 0; a < CT / 2; ++a) acc[a][i] = fma2(S[2 * pc][a], w.x, acc[a][i]);
#pragma unroll
      for (int a = 0; a < CT / 2; ++a) acc[a][i] = fma2(S[2 * pc + 1][a], w.y, acc[a][i]);
    }
#pragma unroll
  for (int i = 0; i < kBlkTok; ++i) {
    float f[CT];
#pragma unroll
    for (int a = 0; a < CT / 2; ++a) unpack2(acc[a][i], f[2 * a], f[2 * a + 1]);
    if (CT == 8) {
#pragma unroll
      for (int a = 0; a < 4; ++a) f[a] += __shfl_xor_sync(0xffffffffu, f[(a + 4) % CT], 4);
#pragma unroll
      for (int a = 0; a < 2; ++a) f[a] += __shfl_xor_sync(0xffffffffu, f[a + 2], 2);
      r[i] = f[0] + __shfl_xor_sync(0xffffffffu, f[1], 1);
    } else {
#pragma unroll
      for (int a = 0; a < 2; ++a) f[a] += __shfl_xor_sync(0xffffffffu, f[a + 2], 4);
      f[0] += __shfl_xor_sync(0xffffffffu, f[1], 2);
      r[i] = f[0] + __shfl_xor_sync(0xffffffffu, f[0], 1);
    }
  }
}

// shared memory of a block: the inputs of four chunks (three on their way) and the prepared vectors of two
template <int DP, int COLS>
struct BlkSmem {
  struct In {
    float raw[kBlkTok][3][DP];                 // k, q, decay (when per channel)
    float v[kBlkTok][COLS];
    float beta[kBlkTok], g[kBlkTok];
  } in[4];
  struct Vec {
    float2 k[kBlkTok][DP], q[kBlkTok][DP], h[kBlkTok][DP], c[DP];      // c_i k_i, c_i q_i, G(4,i) k_i, c_4, every value twice
    float gram[kBlkWarps][16];                 // k_i . G k_j for j < i: index i (i - 1) / 2 + j; q_i . G k_j for j <= i: 6 + i (i + 1) / 2 + j
  } vec[2];
};

template <int PIECES, int CT, bool DELTA, bool WIDE>      // 16 PIECES padded rows (64 or 128); WIDE: 16-byte loads of q, k, decay
__global__ void __launch_bounds__(32 * kBlkWarps, PIECES * CT == 64 ? 4 : 6)
delta_scan_blk_kernel(const float* __restrict__ qkv, long sq, int col_k, int col_v, const float* __restrict__ beta,
                      const float* __restrict__ decay, float* __restrict__ state, float* __restrict__ o, const int* __restrict__ cu,
                      const int* __restrict__ start, const int* __restrict__ state_slot, int heads, int kv_heads, int D, int Dv,
                      int per_channel) {
  constexpr int DP = 16 * PIECES, COLS = 4 * CT * kBlkWarps, NT = 32 * kBlkWarps, PER = DP / NT;      // PER: vector entries a thread prepares
  using Sm = BlkSmem<DP, COLS>;
  extern __shared__ __align__(16) unsigned char blk_smem[];
  Sm& sm = *reinterpret_cast<Sm*>(blk_smem);
  // Entry by entry: the blocks of one portion lie side by side and go to SMs of their own.  With the entry varying fastest a long portion among 15
  // single tokens kept every sixteenth block, two to three to an SM: 2000 tokens, 16 heads of 128 x 128, 2269 us, 1816 in this order.
  const unsigned parts = (Dv + COLS - 1) / COLS, eh = blockIdx.x / parts;
  const int e = static_cast<int>(eh / heads), h = static_cast<int>(eh % heads), g = h / (heads / kv_heads);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rg = lane & 7, x = CT == 8 ? rg : rg >> 1;
  const int cb0 = static_cast<int>(blockIdx.x % parts) * COLS, cw = warp * 4 * CT + (lane >> 3) * CT, c0 = cb0 + cw;      // first column: block, group in it, group
  float* gS = state + (static_cast<long>(state_slot[e]) * heads + h) * D * Dv;
  const bool carried = start[e] > 0;
  const int t0 = cu[e], t1 = cu[e + 1];
  const int nd = per_channel ? heads * D : heads;

  // inputs of the chunk that begins at token t; behind the last token: k = q = v = beta = 0, decay 1
  auto fetch = [&](int t, typename Sm::In& in) {
    constexpr int kLanes = DP / 4, kRows = NT / kLanes;          // a warp (128 rows) or half a warp (64) per (token, vector)
    const int d = (tid % kLanes) * 4;
#pragma unroll
    for (int s = 0; s < 3 * kBlkTok / kRows; ++s) {
      const int row = s * kRows + tid / kLanes, i = (row * 11) >> 5, part = row - 3 * i;       // row / 3 for rows below 12
      if (part == 2 && !per_channel) continue;
      float* dst = &in.raw[i][part][d];
      const float* src = part < 2 ? qkv + static_cast<long>(t + i) * sq + (part == 0 ? col_k : 0) + g * D + d
                                  : decay + static_cast<long>(t + i) * nd + h * D + d;
      const float fill = part < 2 ? 0.f : 1.f;
      if (WIDE) {
        if (t + i < t1 && d < D) cp_async_f32x4(dst, src);
        else *reinterpret_cast<float4*>(dst) = make_float4(fill, fill, fill, fill);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (t + i < t1 && d + j < D) cp_async_f32(dst + j, src + j);
          else dst[j] = fill;
        }
      }
    }
#pragma unroll
    for (int s = 0; s < kBlkTok * COLS / NT; ++s) {
      const int i = (s * NT + tid) / COLS, c = (s * NT + tid) % COLS;
      if (t + i < t1 && cb0 + c < Dv) cp_async_f32(&in.v[i][c], qkv + static_cast<long>(t + i) * sq + col_v + h * Dv + cb0 + c);
      else in.v[i][c] = 0.f;
    }
    if (tid < kBlkTok) {
      if (DELTA && t + tid < t1) cp_async_f32(&in.beta[tid], beta + static_cast<long>(t + tid) * heads + h);
      else in.beta[tid] = 0.f;
    } else if (tid < 2 * kBlkTok && !per_channel) {
      const int i = tid - kBlkTok;
      if (t + i < t1) cp_async_f32(&in.g[i], decay + static_cast<long>(t + i) * nd + h);
      else in.g[i] = 1.f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto prepare = [&](const typename Sm::In& in, typename Sm::Vec& vec) {
    float dots[16] = {};
#pragma unroll
    for (int s = 0; s < PER; ++s) {
      const int d = tid + s * NT;
      float w[kBlkTok], c = 1.f;
#pragma unroll
      for (int i = 0; i < kBlkTok; ++i) {
        const float ki = in.raw[i][0][d], qi = in.raw[i][1][d], gi = per_channel ? in.raw[i][2][d] : in.g[i];
        c *= gi;
#pragma unroll
        for (int j = 0; j < i; ++j) {
          w[j] *= gi;
          if (DELTA) dots[i * (i - 1) / 2 + j] += ki * w[j];
          dots[6 + i * (i + 1) / 2 + j] += qi * w[j];
        }
        w[i] = ki;
        dots[6 + i * (i + 1) / 2 + i] += qi * ki;
        if (DELTA) vec.k[i][d] = make_float2(c * ki, c * ki);
        vec.q[i][d] = make_float2(c * qi, c * qi);
      }
#pragma unroll
      for (int i = 0; i < kBlkTok; ++i) vec.h[i][d] = make_float2(w[i], w[i]);
      vec.c[d] = make_float2(c, c);
    }
    // sixteen sums over the warp: halves are exchanged, lane l ends with entry l >> 1
#pragma unroll
    for (int m = 8; m >= 1; m >>= 1)
#pragma unroll
      for (int a = 0; a < m; ++a) {
        const bool up = (lane & (2 * m)) != 0;
        const float keep = up ? dots[a + m] : dots[a], send = up ? dots[a] : dots[a + m];
        dots[a] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * m);
      }
    dots[0] += __shfl_xor_sync(0xffffffffu, dots[0], 1);
    if ((lane & 1) == 0) vec.gram[warp][lane >> 1] = dots[0];
  };

  if (t0 < t1) {
    fetch(t0, sm.in[0]);
    fetch(t0 + kBlkTok, sm.in[1]);
    fetch(t0 + 2 * kBlkTok, sm.in[2]);
  }
  f32x2 S[2 * PIECES][CT / 2];
#pragma unroll
  for (int r = 0; r < 2 * PIECES; ++r)
#pragma unroll
    for (int a = 0; a < CT / 2; ++a) {
      const int d = (r >> 1) * 16 + rg * 2 + (r & 1), ca = c0 + ((2 * a) ^ x), cb = c0 + ((2 * a + 1) ^ x);
      const bool ok = carried && d < D;
      S[r][a] = pack2(ok && ca < Dv ? gS[static_cast<long>(d) * Dv + ca] : 0.f, ok && cb < Dv ? gS[static_cast<long>(d) * Dv + cb] : 0.f);
    }
  if (t0 < t1) {
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncthreads();
    prepare(sm.in[0], sm.vec[0]);
  }
  const int c_own = c0 + x;
  for (int t = t0, n = 0; t < t1; t += kBlkTok, ++n) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");         // this thread's part of chunk n + 1
    __syncthreads();                               // vectors of chunk n and inputs of n + 1 are here; everyone is done with n - 1
    fetch(t + 3 * kBlkTok, sm.in[(n + 3) & 3]);
    prepare(sm.in[(n + 1) & 3], sm.vec[(n + 1) & 1]);
    const typename Sm::Vec& vec = sm.vec[n & 1];
    const typename Sm::In& in = sm.in[n & 3];
    float u[kBlkTok], r[kBlkTok];
#pragma unroll
    for (int i = 0; i < kBlkTok; ++i) u[i] = in.v[i][cw + x];
    if (DELTA) {
      blk_product<PIECES, CT>(S, &vec.k[0][0], rg, r);
#pragma unroll
      for (int i = 0; i < kBlkTok; ++i) {
        float z = u[i] - r[i];
#pragma unroll
        for (int j = 0; j < i; ++j) z -= (vec.gram[0][i * (i - 1) / 2 + j] + vec.gram[1][i * (i - 1) / 2 + j]) * u[j];
        u[i] = in.beta[i] * z;
      }
    }
    blk_product<PIECES, CT>(S, &vec.q[0][0], rg, r);
#pragma unroll
    for (int i = 0; i < kBlkTok; ++i) {
#pragma unroll
      for (int j = 0; j <= i; ++j) r[i] += (vec.gram[0][6 + i * (i + 1) / 2 + j] + vec.gram[1][6 + i * (i + 1) / 2 + j]) * u[j];
      if ((CT == 8 || (rg & 1) == (i >> 1)) && t + i < t1 && c_own < Dv) o[(static_cast<long>(t + i) * heads + h) * Dv + c_own] = r[i];
    }
    // state: the columns' u come from the lanes that own them
#pragma unroll
    for (int pc = 0; pc < PIECES; ++pc) {
      const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&vec.c[pc * 16 + rg * 2]);
#pragma unroll
      for (int a = 0; a < CT / 2; ++a) {
        S[2 * pc][a] = mul2(S[2 * pc][a], w.x);
        S[2 * pc + 1][a] = mul2(S[2 * pc + 1][a], w.y);
      }
    }
#pragma unroll
    for (int i = 0; i < kBlkTok; ++i) {
      f32x2 ua[CT / 2];
#pragma unroll
      for (int a = 0; a < CT / 2; ++a) {
        const int la = (lane & 24) + ((2 * a) ^ x) * (8 / CT), lb = (lane & 24) + ((2 * a + 1) ^ x) * (8 / CT);
        const float ux = __shfl_sync(0xffffffffu, u[i], la), uy = __shfl_sync(0xffffffffu, u[i], lb);
        ua[a] = pack2(ux, uy);
      }
#pragma unroll
      for (int pc = 0; pc < PIECES; ++pc) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&vec.h[i][pc * 16 + rg * 2]);
#pragma unroll
        for (int a = 0; a < CT / 2; ++a) {
          S[2 * pc][a] = fma2(w.x, ua[a], S[2 * pc][a]);
          S[2 * pc + 1][a] = fma2(w.y, ua[a], S[2 * pc + 1][a]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2 * PIECES; ++r)
#pragma unroll
    for (int a = 0; a < CT / 2; ++a) {
      const int d = (r >> 1) * 16 + rg * 2 + (r & 1), ca = c0 + ((2 * a) ^ x), cb = c0 + ((2 * a + 1) ^ x);
      float fa, fb;
      unpack2(S[r][a], fa, fb);
      if (d < D && ca < Dv) gS[static_cast<long>(d) * Dv + ca] = fa;
      if (d < D && cb < Dv) gS[static_cast<long>(d) * Dv + cb] = fb;
    }
}

template <int PIECES, int CT, bool DELTA, bool WIDE>
cudaError_t launch_delta_blk(dim3 grid, const float* qkv, long sq, int col_k, int col_v, const float* beta, const float* decay, float* state,
                             float* o, const int* cu, const int* start, const int* state_slot, int heads, int kv_heads, int D, int Dv,
                             int per_channel, cudaStream_t s) {
  auto kern = delta_scan_blk_kernel<PIECES, CT, DELTA, WIDE>;
  constexpr int smem = sizeof(BlkSmem<16 * PIECES, 4 * CT * kBlkWarps>);
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  kern<<<grid, 32 * kBlkWarps, smem, s>>>(qkv, sq, col_k, col_v, beta, decay, state, o, cu, start, state_slot, heads, kv_heads, D, Dv, per_channel);
  return cudaGetLastError();
}

// template sizes and block size of the column-resident kernels for a state of `rows` x `cols`; false when they do not fit
bool pick_col_layout(int cols, int rows, int* rows_t, int* split_out, int* threads_out) {
  if (rows > 128 || cols < 1 || cols > 256) return false;
  const int rt = rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128;
  const int split = rt == 128 && cols <= 128 ? 2 : 1;      // 128 rows: two threads per column when the block allows
  int threads = ((cols * split + 31) / 32) * 32;
  if (threads < col_min_threads(rt)) threads = col_min_threads(rt);
  *rows_t = rt;
  *split_out = split;
  *threads_out = threads;
  return true;
}
bool col_form_fits(int cols, int rows) {
  int rows_t, split, threads;
  return pick_col_layout(cols, rows, &rows_t, &split, &threads);
}

// rows per thread / row groups for a state of `rows` x `cols`: as many row groups as 512 threads allow (256 when a thread
// holds 64 rows), at most 64 rows per thread, and enough threads to fetch a token's inputs with kPre loads each
bool pick_reg_layout(int cols, int rows, int per_token, int* R_out, int* rpt_out, int* threads_out) {
  if (cols > 512) return false;
  int R = 512 / cols;
  if (R > rows) R = rows;
  if (R < 1) return false;
  int need = (rows + R - 1) / R;
  if (need > 32) {
    R = 256 / cols;
    if (R > rows) R = rows;
    if (R < 1) return false;
    need = (rows + R - 1) / R;
    if (need > 64) return false;
    if (need <= 32) need = 33;                      // stays in the 64-row variant, whose blocks have 256 threads
  }
  const int rpt = need <= 4 ? 4 : need <= 8 ? 8 : need <= 16 ? 16 : need <= 32 ? 32 : 64;
  int threads = ((cols * R + 31) / 32) * 32;
  const int for_loads = (((per_token + kPre - 1) / kPre + 31) / 32) * 32;
  if (threads < for_loads) threads = for_loads;
  if (threads > (rpt == 64 ? 256 : 512)) return false;
  *R_out = R; *rpt_out = rpt; *threads_out = threads;
  return true;
}

int pick_rows(int cols, int rows) {
  // threads = cols * R <= 512, R <= rows
  int R = 512 / cols;
  if (R < 1) R = 1;
  if (R > rows) R = rows;
  if (R > 16) R = 16;
  return R;
}

// ---------------------------------------------------------------------------------------------------------------------
// Matrix memory with exponential gates and a running maximum (mLSTM).  Per head, with log gates i and f of the token and the
// carried maximum m (0 for a new sequence):  m' = max(f + m, i);  S = exp(f + m - m') S + exp(i - m') k v^T  and the
// normaliser n likewise with k alone.  n is kept as one more column of the state (a value that is always 1), so the state
// of a head is [D, Dv + 1] and its read-out S^T q gives the numerator in columns 0 .. Dv-1 and n . q in column Dv; the division
// is left to nrl_mlstm_out.  The raw gates are capped (cap * tanh(z / cap), cap > 0) and the forget gate goes through
// log-sigmoid.  Block per (entry, head): thread c keeps column c of the state in ROWS registers; one more warp forms the
// gates of the next token while the columns work on the current one (the recurrence of m is one dependent chain per head).
// ---------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float logsigmoid_(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

struct MlstmGate {
  float a, b, m;
};
__device__ __forceinline__ MlstmGate mlstm_gate(float i_raw, float f_raw, float cap, float m_prev) {
  const float ig = cap > 0.f ? cap * tanhf(i_raw / cap) : i_raw;
  const float fg = logsigmoid_(cap > 0.f ? cap * tanhf(f_raw / cap) : f_raw);
  MlstmGate g;
  g.m = fmaxf(fg + m_prev, ig);
  g.a = expf(fg + m_prev - g.m);
  g.b = expf(ig - g.m);
  return g;
}

// SPLIT (1 or 2) threads share a column as in the other column-resident scans (ColStage): neighbouring lanes hold the upper and
// the lower half of its rows and add their partial sums with one shuffle.
template <int ROWS, int SPLIT>
__global__ void __launch_bounds__(ROWS >= 128 ? 320 : ROWS >= 64 ? 256 : 544)      // 128 rows: 168 registers, two blocks of 192 threads per SM
mlstm_scan_col_kernel(const float* __restrict__ qkv, long sq, int col_q, int col_k, int col_v, int col_i, int col_f,
                      const float* __restrict__ i_bias, const float* __restrict__ f_bias, float cap, float q_scale,
                      float* __restrict__ state, float* __restrict__ mstate, float* __restrict__ o, float* __restrict__ m_out,
                      const int* __restrict__ cu, const int* __restrict__ start, const int* __restrict__ state_slot, int heads, int D,
                      int Dv, int Cs) {
  using St = ColStage<ROWS, SPLIT>;
  constexpr int RH = St::RH, VL = St::VL, L = 2 * VL + 4;  // per token: q | k | a, b
  constexpr int kStagePre = (2 * ROWS + 63) / 64;          // a block has at least 64 threads
  __shared__ __align__(16) float stage[2 * L];
  const int e = blockIdx.x, h = blockIdx.y;
  const int tid = threadIdx.x, nth = blockDim.x, ncol = nth - 32, C = Dv + 1;        // ncol threads own columns, the last warp the gates
  const int c = tid / SPLIT, half = tid % SPLIT, r0 = half * RH;
  const bool gate_lane = tid == ncol, col_thread = tid < ncol, live = col_thread && c < C;
  const long slot = state_slot[e];
  float* gS = state + (slot * heads + h) * D * Cs;       // rows of Cs >= Dv + 1 floats
  const bool carried = start[e] > 0;
  float S[RH];
#pragma unroll
  for (int i = 0; i < RH; ++i) S[i] = (live && r0 + i < D && carried) ? gS[static_cast<long>(r0 + i) * Cs + c] : 0.f;
  const int t0 = cu[e], t1 = cu[e + 1];
  const float ib = i_bias != nullptr ? i_bias[h] : 0.f, fb = f_bias != nullptr ? f_bias[h] : 0.f;
  float m_run = carried ? mstate[slot * heads + h] : 0.f;
  MlstmGate gt = {0.f, 0.f, 0.f};
  float pre[kStagePre], pre_v = 0.f;
  auto fetch = [&](int t) {
    const float* row = qkv + static_cast<long>(t) * sq;
#pragma unroll
    for (int i = 0; i < kStagePre; ++i) {
      const int idx = tid + i * nth;
      if (idx < 2 * ROWS) {
        const int d = idx < ROWS ? idx : idx - ROWS;
        pre[i] = d < D ? (idx < ROWS ? row[col_q + h * D + d] * q_scale : row[col_k + h * D + d]) : 0.f;
      }
    }
    if (col_thread) pre_v = c < Dv ? row[col_v + h * Dv + c] : 1.f;
    if (gate_lane) {
      gt = mlstm_gate(row[col_i + h] + ib, row[col_f + h] + fb, cap, m_run);
      m_run = gt.m;
    }
  };
  if (t0 < t1) fetch(t0);
  for (int t = t0; t < t1; ++t) {
    float* v = stage + ((t - t0) & 1) * L;
#pragma unroll
    for (int i = 0; i < kStagePre; ++i) {
      const int idx = tid + i * nth;
      if (idx < 2 * ROWS) v[(idx < ROWS ? 0 : VL) + St::at(idx < ROWS ? idx : idx - ROWS)] = pre[i];
    }
    if (gate_lane) {
      v[2 * VL] = gt.a;
      v[2 * VL + 1] = gt.b;
      m_out[static_cast<long>(t) * heads + h] = gt.m;
    }
    const float v_cur = pre_v;
    __syncthreads();
    if (t + 1 < t1) fetch(t + 1);
    if (col_thread) {
      const float a = v[2 * VL], bv = v[2 * VL + 1] * v_cur;
      const float4* vq = reinterpret_cast<const float4*>(v + half * (RH + 4));
      const float4* vk = reinterpret_cast<const float4*>(v + VL + half * (RH + 4));
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < RH / 4; ++i) {
        const float4 kk = vk[i], qq = vq[i];
        S[4 * i] = a * S[4 * i] + kk.x * bv;
        S[4 * i + 1] = a * S[4 * i + 1] + kk.y * bv;
        S[4 * i + 2] = a * S[4 * i + 2] + kk.z * bv;
        S[4 * i + 3] = a * S[4 * i + 3] + kk.w * bv;
        acc[0] += S[4 * i] * qq.x;
        acc[1] += S[4 * i + 1] * qq.y;
        acc[2] += S[4 * i + 2] * qq.z;
        acc[3] += S[4 * i + 3] * qq.w;
      }
      float tot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
      if (SPLIT == 2) tot += __shfl_xor_sync(0xffffffffu, tot, 1);
      if (live && half == 0) o[(static_cast<long>(t) * heads + h) * C + c] = tot;
    }
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RH; ++i)
      if (r0 + i < D) gS[static_cast<long>(r0 + i) * Cs + c] = S[i];
  }
  if (gate_lane && t0 < t1) mstate[slot * heads + h] = m_run;
}

// Any size: the state stays in global memory, thread per column, every thread forms the gates itself.
__global__ void mlstm_scan_kernel(const float* __restrict__ qkv, long sq, int col_q, int col_k, int col_v, int col_i, int col_f,
                                  const float* __restrict__ i_bias, const float* __restrict__ f_bias, float cap, float q_scale,
                                  float* __restrict__ state, float* __restrict__ mstate, float* __restrict__ o, float* __restrict__ m_out,
                                  const int* __restrict__ cu, const int* __restrict__ start, const int* __restrict__ state_slot, int heads,
                                  int D, int Dv, int Cs) {
  const int e = blockIdx.x, h = blockIdx.y, C = Dv + 1;
  const long slot = state_slot[e];
  float* gS = state + (slot * heads + h) * D * Cs;
  const bool carried = start[e] > 0;
  const float ib = i_bias != nullptr ? i_bias[h] : 0.f, fb = f_bias != nullptr ? f_bias[h] : 0.f;
  const float m0 = carried ? mstate[slot * heads + h] : 0.f;
  __syncthreads();                                         // every thread has read the carried maximum before thread 0 replaces it
  const int t0 = cu[e], t1 = cu[e + 1];
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float m_run = m0;
    for (int t = t0; t < t1; ++t) {
      const float* row = qkv + static_cast<long>(t) * sq;
      const MlstmGate gt = mlstm_gate(row[col_i + h] + ib, row[col_f + h] + fb, cap, m_run);
      m_run = gt.m;
      const float bv = gt.b * (c < Dv ? row[col_v + h * Dv + c] : 1.f);
      float acc = 0.f;
      for (int d = 0; d < D; ++d) {
        const float old = (carried || t > t0) ? gS[static_cast<long>(d) * Cs + c] : 0.f;
        const float sv = gt.a * old + row[col_k + h * D + d] * bv;
        gS[static_cast<long>(d) * Cs + c] = sv;
        acc += sv * (row[col_q + h * D + d] * q_scale);
      }
      o[(static_cast<long>(t) * heads + h) * C + c] = acc;
      if (c == 0) m_out[static_cast<long>(t) * heads + h] = gt.m;
    }
    if (c == 0 && t0 < t1) mstate[slot * heads + h] = m_run;
  }
}

// warp per (token, head): y = o[:Dv] / (max(|o[Dv]|, exp(-m)) + 1e-6); out = scale * y / rms(y) * w * sigmoid(gate)
template <typename OT>
__global__ void mlstm_out_kernel(const float* __restrict__ o, const float* __restrict__ m, const float* __restrict__ gate, long sg,
                                 const float* __restrict__ w, float eps, float scale, OT* __restrict__ out, long so, long T, int heads,
                                 int Dv) {
  const long wid = (blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= T * heads) return;
  const long t = wid / heads;
  const int h = static_cast<int>(wid - t * heads);
  const float* row = o + wid * (Dv + 1);
  const float inv = 1.f / (fmaxf(fabsf(row[Dv]), expf(-m[wid])) + 1e-6f);
  float ss = 0.f;
  for (int c = lane; c < Dv; c += 32) {
    const float y = row[c] * inv;
    ss += y * y;
  }
  ss = warp_sum(ss);
  const float r = 1.f / sqrtf(ss / static_cast<float>(Dv) + eps);
  for (int c = lane; c < Dv; c += 32) {
    const long col = static_cast<long>(h) * Dv + c;
    const float g = gate[t * sg + col];
    const float val = scale * (row[c] * inv * r * w[col] * (1.f / (1.f + expf(-g))));
    if constexpr (sizeof(OT) == 4) out[t * so + col] = val;
    else out[t * so + col] = __float2bfloat16_rn(val);
  }
}

}  // namespace

extern "C" {

cudaError_t nrl_causal_conv(const float* in, long si, const float* in_bias, int act, const float* w, const float* bias,
                            const float* state, float* out, long so, const int* cu, const int* tok_entry, const int* start,
                            const int* state_slot, int T, int E, int C, int taps, cudaStream_t s) {
  if (T <= 0 || C <= 0) return cudaSuccess;
  if (taps < 1 || taps > kMaxTaps) return cudaErrorInvalidValue;
  if (T >= 2 * kConvTok && T >= 2 * E && (T + kConvTok - 1) / kConvTok <= 65535) {     // prompt portions: runs of tokens per thread
    const dim3 grid((C + 127) / 128, (T + kConvTok - 1) / kConvTok);
    if (taps <= 4)
      causal_conv_run_kernel<4><<<grid, 128, 0, s>>>(in, si, in_bias, act, w, bias, state, out, so, cu, tok_entry, start, state_slot, T, C, taps);
    else
      causal_conv_run_kernel<kMaxTaps><<<grid, 128, 0, s>>>(in, si, in_bias, act, w, bias, state, out, so, cu, tok_entry, start, state_slot, T, C, taps);
    return cudaGetLastError();
  }
  const long n = static_cast<long>(T) * C;
  causal_conv_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(in, si, in_bias, act, w, bias, state, out, so, cu,
                                                                           tok_entry, start, state_slot, T, C, taps);
  return cudaGetLastError();
}

cudaError_t nrl_causal_conv_carry(const float* in, long si, const float* in_bias, float* state, const int* cu, const int* start,
                                  const int* state_slot, int E, int C, int taps, cudaStream_t s) {
  if (E <= 0 || C <= 0 || taps <= 1) return cudaSuccess;
  if (taps > kMaxTaps) return cudaErrorInvalidValue;
  const long n = static_cast<long>(E) * C;
  causal_conv_carry_kernel<<<static_cast<unsigned>((n + 127) / 128), 128, 0, s>>>(in, si, in_bias, state, cu, start, state_slot, E, C, taps);
  return cudaGetLastError();
}

cudaError_t nrl_ssd_scan(const float* xbc, long sx, int col_b, int col_c, const float* dt_raw, long sd, const float* dt_bias,
                         const float* A_log, const float* Dskip, float* state, float* y, const int* cu, const int* start,
                         const int* state_slot, int E, int heads, int groups, int N, int P, int impl, cudaStream_t s) {
  if (E <= 0) return cudaSuccess;
  if (P > 512 || heads % groups != 0 || impl < 0 || impl > 3) return cudaErrorInvalidValue;
  if (impl == 0 || impl == 1) {
    int rt, split, threads;
    if (pick_col_layout(P, N, &rt, &split, &threads)) {
#define NRL_SSDC(R_, S_)                                                                                                           \
  if (rt == R_ && split == S_) {                                                                                                   \
    ssd_scan_col_kernel<R_, S_><<<dim3(E, heads), threads, 0, s>>>(xbc, sx, col_b, col_c, dt_raw, sd, dt_bias, A_log, Dskip, state, y, \
                                                                   cu, start, state_slot, heads, groups, N, P);                    \
    return cudaGetLastError();                                                                                                     \
  }
      NRL_SSDC(16, 1) NRL_SSDC(32, 1) NRL_SSDC(64, 1) NRL_SSDC(128, 1) NRL_SSDC(128, 2)
#undef NRL_SSDC
    }
    if (impl == 1) return cudaErrorInvalidValue;
  }
  if (impl != 3) {
    int R, rpt, threads;
    const size_t smem_reg = sizeof(float) * (2 * (2 * static_cast<size_t>(N) + P) + 512);
    if (pick_reg_layout(P, N, 2 * N + P, &R, &rpt, &threads) && smem_reg <= 48 * 1024) {
      const size_t smem = sizeof(float) * (2 * (2 * static_cast<size_t>(N) + P) + static_cast<size_t>(R) * P);
#define NRL_SSD(RPT_)                                                                                                              \
  if (rpt == RPT_) {                                                                                                               \
    ssd_scan_reg_kernel<RPT_><<<dim3(E, heads), threads, smem, s>>>(xbc, sx, col_b, col_c, dt_raw, sd, dt_bias, A_log, Dskip, state, y, \
                                                                    cu, start, state_slot, heads, groups, N, P, R);                \
    return cudaGetLastError();                                                                                                     \
  }
      NRL_SSD(4) NRL_SSD(8) NRL_SSD(16) NRL_SSD(32) NRL_SSD(64)
#undef NRL_SSD
    }
    if (impl == 2) return cudaErrorInvalidValue;
  }
  const int R = pick_rows(P, N);
  const int threads = ((P * R + 31) / 32) * 32;
  const size_t smem = sizeof(float) * (static_cast<size_t>(N) * P + 2 * N + P + static_cast<size_t>(R) * P);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(ssd_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    configured = 200 * 1024;
  }
  ssd_scan_kernel<<<dim3(E, heads), threads, smem, s>>>(xbc, sx, col_b, col_c, dt_raw, sd, dt_bias, A_log, Dskip, state, y, cu, start,
                                                        state_slot, heads, groups, N, P, R);
  return cudaGetLastError();
}

cudaError_t nrl_delta_prep(float* qkv, long sq, int col_k, const float* b_raw, long sb, const float* a_raw, long sa,
                           const float* dt_bias, const float* A_log, float* beta, float* decay, int T, int heads, int kv_heads, int D,
                           int per_channel, cudaStream_t s) {
  if (T <= 0) return cudaSuccess;
  delta_prep_kernel<<<T, 128, 0, s>>>(qkv, sq, col_k, b_raw, sb, a_raw, sa, dt_bias, A_log, beta, decay, heads, kv_heads, D,
                                      per_channel);
  return cudaGetLastError();
}

cudaError_t nrl_gla_prep(float* qkv, long sq, const float* a_raw, long sa, const float* a_bias, float tau, float* decay, int T,
                         int heads, int D, cudaStream_t s) {
  if (T <= 0) return cudaSuccess;
  if (!(tau > 0.f)) return cudaErrorInvalidValue;
  gla_prep_kernel<<<T, 128, 0, s>>>(qkv, sq, a_raw, sa, a_bias, 1.f / tau, decay, heads * D, D);
  return cudaGetLastError();
}

// Other steps of prompt portions (a decay per key channel above all) take four tokens at a time.  Where the column-resident form fits (Dv <= 256) the lines are
//   D > 32      a smaller state is padded to 64 rows here, to 16 or 32 there: 64 entries of 128 tokens, 16 heads of 32 x 32, 230 us against 83; one
//               row more, 33 x 33, 237 / 316
//   T >= 20 E   a thread's state is not read in whole lines, so that short portions pay more for it: 128 x 128, 64 entries of 2: 95 us against 50,
//               of 4: 97 / 65; 16 entries of 12: 38 / 38, 8 of 16: 30 / 26, 16 of 20: 45 / 54; 64 x 128, 16 of 16: 26 / 24, of 20: 30 / 30.
// Above: 16 entries of 2048, 128 x 128: 2300 / 4350, one of 2000: 1515 / 2119; 64 x 64, 16 of 1000: 689 / 1013; without the delta (beta == nullptr) 0.4 to 0.9
// of the other's time; single tokens beside one portion of 2000, 128 x 128: 15 of them 1816 / 2143, 64 1909 / 2171.  Where the column form does not fit
// (Dv > 256) the row groups take 1.1 to 10 times as long from twelve tokens an entry on, at D = 16 to 128.
int nrl_delta_scan_blocked(long E, long T, int D, int Dv) {
  return D <= 128 && (col_form_fits(Dv, D) ? D > 32 && T >= 20 * E : T >= 12 * E);
}

// One decay per head and rows of q, k and v on 16-byte boundaries: 32 tokens at a time on the tensor cores (delta_chunk_tc.cu), where a block has an SM to itself
// and starts with 64 KB of state, so that short portions need a full state and many portions need more tokens each.  us there / the better of the others,
// 16 heads (E x heads blocks; one to a block of 128 columns):
//   any state, blocks <= SMs, T >= 20 E   1 x 20 tokens 64 x 64: 14 / 15, 128 x 128: 15 / 23; 1 x 2000, 128 x 128: 310 / 1450
//   128 x 128, T >= 20 E                  16 x 20: 29 / 43; 64 x 20: 99 / 156; 16 x 2048: 630 / 2290; 64 single tokens beside a portion of 2000 take the same line
//   64 x 128, T >= 32 E                   256 x 20: 293 / 264, x 32: 305 / 345
//   128 x 64 (half the lanes), T >= 48 E  256 x 20: 366 / 285, x 32: 375 / 377, x 48: 517 / 497; 32 x 48: 75 / 72, x 64: 74 / 93
//   64 x 64, T >= 128 E                   256 x 64: 445 / 331; 128 x 96: 285 / 265, x 128: 343 / 343; 64 x 128: 190 / 235
// Rows that are not aligned come float by float: 64 x 256 tokens, 33 x 33: 531 / 456; they stay with four tokens at a time.
int nrl_delta_scan_chunked(long E, long T, int heads, int D, int Dv, int num_sms) {
  if (D <= 32 || D > 128 || T < 20 * E) return 0;
  if (E * heads * ((Dv + 127) / 128) <= num_sms) return 1;
  return T >= (Dv > 64 ? (D > 64 ? 20 : 32) : (D > 64 ? 48 : 128)) * E;
}

static bool delta_rows16(const float* qkv, long sq, int col_k, int col_v, int D, int Dv) {
  return D % 4 == 0 && Dv % 4 == 0 && sq % 4 == 0 && col_k % 4 == 0 && col_v % 4 == 0 && reinterpret_cast<uintptr_t>(qkv) % 16 == 0;
}
static bool delta_takes_chunks(bool rows16, long E, long T, int heads, int D, int Dv, int per_channel, int impl, int num_sms) {
  return !per_channel && D >= 1 && D <= 128 && Dv >= 1 && (impl >= 5 || (impl == 0 && rows16 && nrl_delta_scan_chunked(E, T, heads, D, Dv, num_sms)));
}
// Blocks share the chunks of all items (delta_chunk_tc.cu) where rounds of whole items leave many SMs without one in the last: a chunk costs an eighth more
// there, and starting anew between segments about four chunks, so it comes into question for a gain of a tenth by that estimate with entries of equal lengths, for
// which the gain is largest; the lengths decide (nrl_delta_line_mode).  us, items whole / shared (entries of tokens, 16 heads): 128 x 128, 10 of 2048 625 / 381,
// 12 of 700 228 / 210; 64 x 64, 11 of 300 98 / 88; not taken: 16 of 2048 630 / 617, 32 of 1000 647 / 688, 16 of 256 98 / 121, 64 of 200 309 / 318.
static bool delta_line_fits(long E, long T, int heads, int Dv) {
  return E <= 4096 && T / 32 + E < (1l << 30) / (heads * ((Dv + 127) / 128));
}
int nrl_delta_scan_shared(long E, long T, int heads, int Dv, int num_sms) {
  const long items = E * heads * ((Dv + 127) / 128), rounds = (items + num_sms - 1) / num_sms;
  if (items <= num_sms || !delta_line_fits(E, T, heads, Dv)) return 0;
  const double chunks = static_cast<double>(T) / (32.0 * E);
  return 1.13 * items * chunks / num_sms + 4.0 < 0.9 * rounds * chunks;
}
int nrl_delta_line_mode(const long* tokens, long E, long T, int heads, int Dv, int impl, int num_sms) {
  if (impl == 6) return delta_line_fits(E, T, heads, Dv) ? 2 : 0;
  if (!nrl_delta_scan_shared(E, T, heads, Dv, num_sms)) return 0;
  return tokens == nullptr ? 1 : nrl_delta_line_pays(tokens, E, heads, Dv, num_sms) ? 2 : 0;
}
long nrl_delta_scan_scratch(const float* qkv, long sq, int col_k, int col_v, long E, long T, int heads, int D, int Dv, int per_channel, int impl, int line, int num_sms) {
  if (line == 0 || E <= 0 || !delta_rows16(qkv, sq, col_k, col_v, D, Dv) || !delta_takes_chunks(true, E, T, heads, D, Dv, per_channel, impl, num_sms)) return 0;
  return nrl_delta_line_bytes(E, heads, Dv, num_sms);
}

cudaError_t nrl_delta_scan(const float* qkv, long sq, int col_k, int col_v, const float* beta, const float* decay, float* state,
                           float* o, const int* cu, const int* start, const int* state_slot, int E, int T, int heads, int kv_heads,
                           int D, int Dv, int per_channel, int impl, int line, int num_sms, void* scratch, cudaStream_t s) {
  if (E <= 0) return cudaSuccess;
  if (Dv > 512 || heads % kv_heads != 0 || impl < 0 || impl > 6 || (impl == 6 && scratch == nullptr)) return cudaErrorInvalidValue;
  const bool rows16 = delta_rows16(qkv, sq, col_k, col_v, D, Dv);
  if (delta_takes_chunks(rows16, E, T, heads, D, Dv, per_channel, impl, num_sms))
    return nrl_delta_chunk_tc(qkv, sq, col_k, col_v, beta, decay, state, o, cu, start, state_slot, E, heads, kv_heads, D, Dv, rows16, scratch, num_sms, line == 2, s);
  if (impl >= 5) return cudaErrorInvalidValue;
  if (D >= 1 && D <= 128 && Dv >= 1 && (impl == 4 || (impl == 0 && nrl_delta_scan_blocked(E, T, D, Dv)))) {
    const bool wide = D % 4 == 0 && sq % 4 == 0 && col_k % 4 == 0 && reinterpret_cast<uintptr_t>(qkv) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(decay) % 16 == 0;
    // eight columns per thread unless that leaves SMs without a block (one entry of 2048, 16 heads: four columns 1564 us, eight 1816; 16 entries:
    // 3730 / 2310)
    const int ct = static_cast<long>(E) * heads * ((Dv + 63) / 64) >= num_sms ? 8 : 4;
    const dim3 grid(static_cast<unsigned>(E) * heads * ((Dv + 8 * ct - 1) / (8 * ct)));
#define NRL_DELTAB(P_, C_, B_)                                                                                                   \
  if ((D <= 64 ? 4 : 8) == P_ && ct == C_ && (beta != nullptr) == B_)                                                              \
    return (wide ? launch_delta_blk<P_, C_, B_, true> : launch_delta_blk<P_, C_, B_, false>)(                                      \
        grid, qkv, sq, col_k, col_v, beta, decay, state, o, cu, start, state_slot, heads, kv_heads, D, Dv, per_channel, s);
    NRL_DELTAB(4, 4, true) NRL_DELTAB(4, 4, false) NRL_DELTAB(4, 8, true) NRL_DELTAB(4, 8, false)
    NRL_DELTAB(8, 4, true) NRL_DELTAB(8, 4, false) NRL_DELTAB(8, 8, true) NRL_DELTAB(8, 8, false)
#undef NRL_DELTAB
  }
  if (impl == 4) return cudaErrorInvalidValue;
  if (impl == 0 || impl == 1) {
    int rt, split, threads;
    if (pick_col_layout(Dv, D, &rt, &split, &threads)) {
#define NRL_DELTAC(R_, S_)                                                                                                         \
  if (rt == R_ && split == S_) {                                                                                                   \
    delta_scan_col_kernel<R_, S_><<<dim3(E, heads), threads, 0, s>>>(qkv, sq, col_k, col_v, beta, decay, state, o, cu, start,        \
                                                                     state_slot, heads, kv_heads, D, Dv, per_channel);             \
    return cudaGetLastError();                                                                                                     \
  }
      NRL_DELTAC(16, 1) NRL_DELTAC(32, 1) NRL_DELTAC(64, 1) NRL_DELTAC(128, 1) NRL_DELTAC(128, 2)
#undef NRL_DELTAC
    }
    if (impl == 1) return cudaErrorInvalidValue;
  }
  if (impl != 3) {
    int R, rpt, threads;
    const size_t smem_reg = sizeof(float) * (6 * static_cast<size_t>(D) + 2 * 512 + 64);
    if (pick_reg_layout(Dv, D, 3 * D, &R, &rpt, &threads) && smem_reg <= 48 * 1024) {
      const size_t smem = sizeof(float) * (6 * static_cast<size_t>(D) + 2 * static_cast<size_t>(R) * Dv + R);
#define NRL_DELTA(RPT_)                                                                                                            \
  if (rpt == RPT_) {                                                                                                               \
    delta_scan_reg_kernel<RPT_><<<dim3(E, heads), threads, smem, s>>>(qkv, sq, col_k, col_v, beta, decay, state, o, cu, start,       \
                                                                      state_slot, heads, kv_heads, D, Dv, per_channel, R);         \
    return cudaGetLastError();                                                                                                     \
  }
      NRL_DELTA(4) NRL_DELTA(8) NRL_DELTA(16) NRL_DELTA(32) NRL_DELTA(64)
#undef NRL_DELTA
    }
    if (impl == 2) return cudaErrorInvalidValue;
  }
  const int R = pick_rows(Dv, D);
  const int threads = ((Dv * R + 31) / 32) * 32;
  const size_t smem = sizeof(float) * (static_cast<size_t>(D) * Dv + 3 * D + 2 * static_cast<size_t>(R) * Dv + 1);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    configured = 200 * 1024;
  }
  delta_scan_kernel<<<dim3(E, heads), threads, smem, s>>>(qkv, sq, col_k, col_v, beta, decay, state, o, cu, start, state_slot, heads,
                                                          kv_heads, D, Dv, per_channel, R);
  return cudaGetLastError();
}

cudaError_t nrl_mlstm_scan(const float* qkv, long sq, int col_q, int col_k, int col_v, int col_i, int col_f, const float* i_bias,
                           const float* f_bias, float cap, float q_scale, float* state, float* mstate, float* o, float* m_out,
                           const int* cu, const int* start, const int* state_slot, int E, int heads, int D, int Dv, int Cs,
                           int single_token, int impl, cudaStream_t s) {
  if (E <= 0) return cudaSuccess;
  if (D < 1 || Dv < 1 || Cs < Dv + 1 || impl < 0 || impl > 2) return cudaErrorInvalidValue;
  // Steps of single tokens only move the state: two threads per column of a 128-row state put more loads in flight.  Entries
  // that hold runs of tokens are bound by the token loop, where one thread per column keeps its rows in registers without spills.
  const int rt = D <= 16 ? 16 : D <= 32 ? 32 : D <= 64 ? 64 : 128;
  const int split = single_token && rt == 128 && (((Dv + 1) * 2 + 31) / 32) * 32 + 32 <= 320 ? 2 : 1;
  const int ncol = (((Dv + 1) * split + 31) / 32) * 32;
  if (impl != 2 && D <= 128 && ncol + 32 <= (rt >= 128 ? 320 : rt >= 64 ? 256 : 544)) {
#define NRL_ML(R_, S_)                                                                                                             \
  mlstm_scan_col_kernel<R_, S_><<<dim3(E, heads), ncol + 32, 0, s>>>(qkv, sq, col_q, col_k, col_v, col_i, col_f, i_bias, f_bias, cap,  \
                                                                     q_scale, state, mstate, o, m_out, cu, start, state_slot, heads, D, Dv, Cs)
    if (rt == 16) NRL_ML(16, 1);
    else if (rt == 32) NRL_ML(32, 1);
    else if (rt == 64) NRL_ML(64, 1);
    else if (split == 2) NRL_ML(128, 2);
    else NRL_ML(128, 1);
#undef NRL_ML
    return cudaGetLastError();
  }
  if (impl == 1) return cudaErrorInvalidValue;
  const int th = Dv + 1 >= 256 ? 256 : ((Dv + 1 + 31) / 32) * 32;
  mlstm_scan_kernel<<<dim3(E, heads), th, 0, s>>>(qkv, sq, col_q, col_k, col_v, col_i, col_f, i_bias, f_bias, cap, q_scale, state, mstate,
                                                  o, m_out, cu, start, state_slot, heads, D, Dv, Cs);
  return cudaGetLastError();
}

cudaError_t nrl_mlstm_out(const float* o, const float* m, const float* gate, long sg, const float* w, float eps, float scale, void* out,
                          long so, int out_f32, int T, int heads, int Dv, cudaStream_t s) {
  if (T <= 0) return cudaSuccess;
  const long warps = static_cast<long>(T) * heads;
  const unsigned blocks = static_cast<unsigned>((warps + 3) / 4);
  if (out_f32) mlstm_out_kernel<float><<<blocks, 128, 0, s>>>(o, m, gate, sg, w, eps, scale, static_cast<float*>(out), so, T, heads, Dv);
  else mlstm_out_kernel<__nv_bfloat16><<<blocks, 128, 0, s>>>(o, m, gate, sg, w, eps, scale, static_cast<__nv_bfloat16*>(out), so, T, heads, Dv);
  return cudaGetLastError();
}

}  // extern "C"
