// Parts of a decode attention's key walk, merged: out = sum_s 2^(m_s - M) o_s / sum_s 2^(m_s - M) l_s, in the order of the parts.
// One block per row and head, launched while the parts are still being formed (launch.h).  Bound by latency: the first parts' values are asked for before
// their maximum is known, eight at a time.  37 sequences x 2 key heads x 6 rows: 5.3 us with a block per key head that took its rows and
// parts one after the other.
#pragma once
#include "common.cuh"

namespace nrl {

constexpr int kMergeD = 128;             // head size == threads
constexpr int kMergeU = 8;               // parts in flight

struct MergeParams {
  const float* part_o;                   // [S, Hkv, splits, 8, D]
  const float* part_ml;                  // [S, Hkv, splits, 8, 2]: maximum (log2 units), sum
  __nv_bfloat16* out;                    // [S, Hq, D]
  int Hq, Hkv, G, splits;
};

NRL_DEVICE void merge_decode_parts(const MergeParams& p) {
  const int seq = blockIdx.x, head = blockIdx.y, kvh = head / p.G, r = head - kvh * p.G, d = threadIdx.x;
  const long base = (static_cast<long>(seq) * p.Hkv + kvh) * p.splits * 8 + r;
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + base;
  const float* po = p.part_o + base * kMergeD + d;
  float o[kMergeU];
#pragma unroll
  for (int u = 0; u < kMergeU; ++u) o[u] = u < p.splits ? po[u * 8 * kMergeD] : 0.f;
  float M = -INFINITY;
  for (int s0 = 0; s0 < p.splits; s0 += kMergeU) {
#pragma unroll
    for (int u = 0; u < kMergeU; ++u)
      if (s0 + u < p.splits) M = fmaxf(M, ml[(s0 + u) * 8].x);
  }
  float L = 0.f, acc = 0.f;
  for (int s0 = 0; s0 < p.splits; s0 += kMergeU) {
    float2 e[kMergeU];
#pragma unroll
    for (int u = 0; u < kMergeU; ++u) {
      const bool ok = s0 + u < p.splits;
      e[u] = ok ? ml[(s0 + u) * 8] : make_float2(-INFINITY, 0.f);
      if (s0 > 0) o[u] = ok ? po[(s0 + u) * 8 * kMergeD] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kMergeU; ++u) {
      if (s0 + u < p.splits) {
        const float c = e[u].x == -INFINITY ? 0.f : exp2f(e[u].x - M);
        L += e[u].y * c;
        acc += o[u] * c;
      }
    }
  }
  p.out[(static_cast<long>(seq) * p.Hq + head) * kMergeD + d] = __float2bfloat16(L > 0.f ? acc / L : 0.f);
}

}  // namespace nrl
