// Building blocks shared by the tcgen05 attention forward kernels: an MMA whose A operand lives in TMEM, packed float32 arithmetic,
// 2^x, and one 128 x 128 block of the online softmax per thread row.
#pragma once
#include "common.cuh"

namespace nrl {

// D[tmem] (+)= A[tmem] * B[smem desc]: A is [128 lanes][K] bf16, two elements per 32-bit column
NRL_DEVICE void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

NRL_DEVICE float ex2_approx(float x) {       // relative error about 2^-22; 2^-inf = 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
NRL_DEVICE uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
NRL_DEVICE void unpack_f32x2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
NRL_DEVICE uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
NRL_DEVICE uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

NRL_DEVICE uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// lo += the pair's first element, hi += its second
NRL_DEVICE void add_bf16x2(uint32_t pair, float& lo, float& hi) {
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tadd.rn.f32.bf16 %0, a, %0;\n\tadd.rn.f32.bf16 %1, b, %1;\n\t}" : "+f"(lo), "+f"(hi) : "r"(pair));
}

// Packed sequences cut into blocks of BM rows, put in order by the number of blocks in front of (or behind) them: how many blocks have
// `level` or more of them, and the n-th sequence that has more than `level` blocks (both by a whole warp).
template <int BM>
NRL_DEVICE int attn_blocks_from(const int* cu, int num_seqs, int level, int lane) {
  int n = 0;
  for (int s = lane; s < num_seqs; s += 32) n += max(0, (cu[s + 1] - cu[s] + BM - 1) / BM - level);
  return __reduce_add_sync(0xffffffffu, n);
}
template <int BM>
NRL_DEVICE int attn_nth_sequence(const int* cu, int num_seqs, int level, int n, int lane) {
  for (int s0 = 0; s0 < num_seqs; s0 += 32) {
    const int s = s0 + lane;
    const bool has = s < num_seqs && (cu[s + 1] - cu[s] + BM - 1) / BM > level;
    const uint32_t m = __ballot_sync(0xffffffffu, has);
    const uint32_t hit = __ballot_sync(0xffffffffu, has && __popc(m & ((1u << lane) - 1)) == n);
    if (hit != 0) return s0 + __ffs(hit) - 1;
    n -= __popc(m);
  }
  return 0;                                    // not reached for n below their number
}

NRL_DEVICE void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
NRL_DEVICE void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
NRL_DEVICE void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// 32-byte global accesses (one full sector per lane); addresses are multiples of 32
NRL_DEVICE void ldg_v8(const float* a, float (&f)[8]) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "l"(a));
}

constexpr int kAtD = 128;                    // head size
constexpr int kAtBN = 128;                   // keys per block
constexpr int kAtPanel = 128 * 128;          // [128 rows][64 x bf16], 128B-swizzled (16 KB)
constexpr int kAtTile = 2 * kAtPanel;        // [128 rows][128 columns] (32 KB)
constexpr int kAtThreads = 384;              // warp 0 TMA, warp 1 MMA (2, 3 helpers); warps 4..7 and 8..11 softmax of tile A and B
// registers: 384 x 168 at launch; the softmax warpgroups take 2 x 128 x 208, the first warpgroup keeps 128 x 88
NRL_DEVICE void attn_regs_softmax() { asm volatile("setmaxnreg.inc.sync.aligned.u32 208;"); }
NRL_DEVICE void attn_regs_issue() { asm volatile("setmaxnreg.dec.sync.aligned.u32 88;"); }
// TMEM columns: S_A | S_B (P overwrites the first 64 columns of its S) | O_A | O_B
constexpr int kAtTmemO = 256;

// S_X = Q_X K^T: both operands K-major in shared memory
NRL_DEVICE void attn_issue_s(uint32_t t_s, uint32_t q_addr, uint32_t k_addr) {
  constexpr uint32_t idesc = make_idesc(128, kAtBN, 1, 1);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    umma_f16(t_s, make_smem_desc_sw128(q_addr + (k >> 2) * kAtPanel + (k & 3) * 32),
             make_smem_desc_sw128(k_addr + (k >> 2) * kAtPanel + (k & 3) * 32), idesc, k != 0 ? 1u : 0u);
}
// O_X (+)= P_X V: P from TMEM, V in place as an MN-major operand; the first `steps` groups of 16 keys
NRL_DEVICE void attn_issue_pv(uint32_t t_o, uint32_t t_p, uint32_t v_addr, bool first, int steps = 8) {
  constexpr uint32_t idesc = make_idesc_bmn(128, kAtD);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (k < steps) umma_f16_ts(t_o, t_p + k * 8, make_smem_desc_sw128_mn(v_addr + k * 16 * 128, kAtPanel), idesc, (first && k == 0) ? 0u : 1u);
}

// scores outside columns [lo, hi] of this block and not below `keep` become -inf (a bit per column)
NRL_DEVICE uint32_t mask_from(int lo) { return lo <= 0 ? 0xffffffffu : lo >= 32 ? 0u : 0xffffffffu << lo; }
NRL_DEVICE void attn_mask_block(uint32_t (&sv)[4][32], int lo, int hi, int keep) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint32_t upto = ~mask_from(hi + 1 - c * 32);
    const uint32_t see = upto & (mask_from(lo - c * 32) | ~mask_from(keep - c * 32));
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (!(see & (1u << i))) sv[c][i] = 0xff800000u;
  }
}

// Thread = one row of S (128 scores in registers, raw; -inf where masked).  Replaces the scores by P = 2^(s * scale - m) in TMEM
// (bf16), updates the running maximum / sum and rescales the row of O when its maximum moved by more than 2^8 (a stale maximum is
// harmless below that: P stays under 256 and the sum is kept in float).  `first`: O holds nothing yet.  `half`: columns 64 and up are all masked
// and their P is not read.
// EXACT, for results that leave no statistic of the sum: the maximum is the row's own in every block, so that its largest weight is
// exactly 1, and the sum adds the weights as P V sees them, rounded.  Error against float64, 16 x 2048 tokens with window 1024: 2.51e-3, lazily
// and with unrounded sums 2.56e-3, mma.sync kernel 2.52e-3; it costs 349 -> 368 us.  (A sum whose logarithm the backward forms P from adds unrounded weights.)
// Neither the tensor pipe nor the special-function unit is saturated while this runs (56 % each, 4 x 4096 tokens): what bounds it is the chain from
// a tile's scores to its P and on to the next scores.  A share of the 2^x on the FMA pipe (polynomial) brought nothing: 430 -> 438 / 454 us with
// 2 / 3 of 8 pairs at 16 x 2048 tokens.
template <bool EXACT>
NRL_DEVICE void attn_softmax_block(uint32_t (&sv)[4][32], float scale, uint32_t t_p, uint32_t t_o, bool first, float& m_run, float& l_run,
                                   bool half = false) {
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < 32; i += 2)
      mx4[(i >> 1) & 3] = fmaxf(mx4[(i >> 1) & 3], fmaxf(__uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1])));
  const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale;
  const bool moved = mx > (EXACT ? m_run : m_run + 8.f);      // false while nothing has been seen (-inf > -inf)
  const float corr = moved ? ex2_approx(m_run - mx) : 1.f;
  m_run = moved ? mx : m_run;
  const float m_sub = m_run == -INFINITY ? 0.f : m_run;       // 2^(-inf - 0) = 0 for a row without keys so far
  const uint64_t sc2 = pack_f32x2(scale, scale), nm2 = pack_f32x2(-m_sub, -m_sub);
  uint64_t sum2[2] = {0, 0};
  float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h == 1 && half) break;
    uint32_t pv[32];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float a, b;
        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[2 * h + c][i]), __uint_as_float(sv[2 * h + c][i + 1])), sc2, nm2), a, b);
        a = ex2_approx(a);
        b = ex2_approx(b);
        pv[c * 16 + i / 2] = pack_bf16x2(a, b);
        if (EXACT) add_bf16x2(pv[c * 16 + i / 2], sum4[(i >> 1) & 1], sum4[2 + ((i >> 1) & 1)]);
        else sum2[(i >> 1) & 1] = add_f32x2(sum2[(i >> 1) & 1], pack_f32x2(a, b));
      }
    tmem_st_32x32b_x32(t_p + h * 32, pv);
  }
  float s0, s1;
  unpack_f32x2(add_f32x2(sum2[0], sum2[1]), s0, s1);
  if (EXACT) {
    s0 = sum4[0] + sum4[1];
    s1 = sum4[2] + sum4[3];
  }
  l_run = l_run * corr + (s0 + s1);
  // the block's S was committed behind the previous P V, so O is current here
  if (__any_sync(0xffffffffu, moved && !first)) {
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
      uint32_t ov[2][32];
      tmem_ld_32x32b_x32(t_o + c * 64, ov[0]);
      tmem_ld_32x32b_x32(t_o + c * 64 + 32, ov[1]);
      tmem_ld_wait();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < 32; ++i) ov[h][i] = __float_as_uint(__uint_as_float(ov[h][i]) * corr);
        tmem_st_32x32b_x32(t_o + c * 64 + h * 32, ov[h]);
      }
    }
  }
  tmem_st_wait();
}

}  // namespace nrl
