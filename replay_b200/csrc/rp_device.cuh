// Device helpers shared by the replay kernels (sm_100a).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "rp_internal.h"

namespace rp {

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11): 10 rounds of two
// 32x32->64 multiplies with a Weyl key schedule.  Counter-based: every
// (key, counter) pair is an independent draw, so any thread can produce the
// uniform of any (replica, node, step) without state.
__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1,
                                              uint32_t c2, uint32_t c3,
                                              uint32_t k0, uint32_t k1,
                                              uint32_t out[4]) {
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    const uint32_t lo0 = 0xD2511F53u * c0;
    const uint32_t hi0 = __umulhi(0xD2511F53u, c0);
    const uint32_t lo1 = 0xCD9E8D57u * c2;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2);
    const uint32_t n0 = hi1 ^ c1 ^ k0;
    const uint32_t n2 = hi0 ^ c3 ^ k1;
    c0 = n0;
    c1 = lo1;
    c2 = n2;
    c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  out[0] = c0;
  out[1] = c1;
  out[2] = c2;
  out[3] = c3;
}

// Same generator with the 10 round keys precomputed (key schedule hoisted
// out of the per-call work): rk[2 i], rk[2 i + 1] are round i's key words.
__device__ __forceinline__ void philox4x32_10_rk(uint32_t c0, uint32_t c1, uint32_t c2,
                                                 uint32_t c3, const uint32_t *rk,
                                                 uint32_t out[4]) {
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    const uint32_t lo0 = 0xD2511F53u * c0;
    const uint32_t hi0 = __umulhi(0xD2511F53u, c0);
    const uint32_t lo1 = 0xCD9E8D57u * c2;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2);
    const uint32_t n0 = hi1 ^ c1 ^ rk[2 * round];
    const uint32_t n2 = hi0 ^ c3 ^ rk[2 * round + 1];
    c0 = n0;
    c1 = lo1;
    c2 = n2;
    c3 = lo0;
  }
  out[0] = c0;
  out[1] = c1;
  out[2] = c2;
  out[3] = c3;
}

// Two independent calls of philox4x32_10_rk on counters (c0, c1, c2, c3a)
// and (c0, c1, c2, c3b), interleaved round by round so that the two
// dependency chains overlap (twice the instruction-level parallelism).
__device__ __forceinline__ void philox4x32_10_rk_x2(uint32_t c0, uint32_t c1, uint32_t c2,
                                                    uint32_t c3a, uint32_t c3b,
                                                    const uint32_t *rk, uint32_t a[4],
                                                    uint32_t b[4]) {
  uint32_t x0 = c0, x1 = c1, x2 = c2, x3 = c3a;
  uint32_t y0 = c0, y1 = c1, y2 = c2, y3 = c3b;
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    const uint32_t xl0 = 0xD2511F53u * x0, xh0 = __umulhi(0xD2511F53u, x0);
    const uint32_t yl0 = 0xD2511F53u * y0, yh0 = __umulhi(0xD2511F53u, y0);
    const uint32_t xl1 = 0xCD9E8D57u * x2, xh1 = __umulhi(0xCD9E8D57u, x2);
    const uint32_t yl1 = 0xCD9E8D57u * y2, yh1 = __umulhi(0xCD9E8D57u, y2);
    const uint32_t k0 = rk[2 * round], k1 = rk[2 * round + 1];
    x0 = xh1 ^ x1 ^ k0;
    y0 = yh1 ^ y1 ^ k0;
    x2 = xh0 ^ x3 ^ k1;
    y2 = yh0 ^ y3 ^ k1;
    x1 = xl1;
    y1 = yl1;
    x3 = xl0;
    y3 = yl0;
  }
  a[0] = x0; a[1] = x1; a[2] = x2; a[3] = x3;
  b[0] = y0; b[1] = y1; b[2] = y2; b[3] = y3;
}

// Uniform on the 24-bit grid ((x >> 8) + 1) * 2^-24, in (0, 1]; exact in
// float, so host and device agree bit for bit.
__device__ __forceinline__ float unit24(uint32_t x) {
  return __fmul_rn(__uint2float_rn((x >> 8) + 1u), 0x1p-24f);
}

// Random stream layout, key = seed, counter = (node, step, c2, c3):
//  * countdown-mode infection (S->E / S->I) uniform of replica r:
//    c2 = r / 4, c3 = 3, output r % 4 on the 24-bit grid; event iff P > u;
//  * flow (E->I, I->R, R->S) uniform of replica r: bit-sliced -- bit k of
//    U_r (k = 0 is 2^-1) is bit r % 32 of output k % 4 of counter
//    (node, step, r / 32, (k / 4) << 4); event iff U_r < floor(p 2^64)
//    over the first 64 bits (flow_events);
//  * geometric-mode infection uniform: top 8 bits bit-sliced on
//    c3 = 4 | j << 4 (c2 = r / 32), low 56 bits on c2 = r, c3 = 12
//    (infect_event);
//  * Bernoulli initial condition: step 0xFFFFFFFF, c2 = r / 4, c3 = 1;
//  * exact-count initial condition (Floyd): node = draw j, step
//    0xFFFFFFFE, c2 = r, c3 = 2 (+ 4 x network index).
constexpr uint32_t kStreamFlow = 0u;    // bit-sliced flow uniforms, c3 = plane/4 << 4
constexpr uint32_t kStreamInit = 1u;
constexpr uint32_t kStreamPick = 2u;
constexpr uint32_t kStreamInfect = 3u;  // scalar infection uniforms
constexpr uint32_t kStepInit = 0xFFFFFFFFu;
constexpr uint32_t kStepPick = 0xFFFFFFFEu;

// 1 - exp(-x) for x >= 0 from correctly rounded multiplies and adds only
// (no FMA contraction): Cody-Waite reduction x = k ln2 + r with ln2 split in
// a 15-bit head and a tail, then the Taylor series of expm1(-r) through
// r^9/9! in Horner form.  Max error about 1 ulp; NaN propagates (the
// reference's p = 1, zero-exposure case), +inf gives 1.
__device__ __forceinline__ float one_minus_exp_neg(float x) {
  if (x != x) return x;
  if (!(x > 0.0f)) return 0.0f;
  if (x >= 87.0f) return 1.0f;
  const float inv_ln2 = 0x1.715476p+0f;
  const float ln2_hi = 0x1.62e4p-1f;
  const float ln2_lo = 0x1.7f7d1cp-20f;
  const int k = __float2int_rz(__fadd_rn(__fmul_rn(x, inv_ln2), 0.5f));
  const float kf = __int2float_rn(k);
  const float r =
      __fsub_rn(__fsub_rn(x, __fmul_rn(kf, ln2_hi)), __fmul_rn(kf, ln2_lo));
  const float y = -r;
  float p = 0x1.71de3ap-19f;
  p = __fadd_rn(__fmul_rn(p, y), 0x1.a01a02p-16f);
  p = __fadd_rn(__fmul_rn(p, y), 0x1.a01a02p-13f);
  p = __fadd_rn(__fmul_rn(p, y), 0x1.6c16c2p-10f);
  p = __fadd_rn(__fmul_rn(p, y), 0x1.111112p-7f);
  p = __fadd_rn(__fmul_rn(p, y), 0x1.555556p-5f);
  p = __fadd_rn(__fmul_rn(p, y), 0x1.555556p-3f);
  p = __fadd_rn(__fmul_rn(p, y), 0.5f);
  const float em1 = __fadd_rn(y, __fmul_rn(__fmul_rn(y, y), p));
  if (k == 0) return -em1;
  const float scale = __int_as_float((127 - k) << 23);
  const float e = __fmul_rn(__fadd_rn(1.0f, em1), scale);
  return __fsub_rn(1.0f, e);
}

// Per-step flow thresholds (FlowThresholds, rp_internal.h) hold
// floor(p 2^64); p >= 1 is a certain event, p <= 0 none.
// Flow events of the replicas selected by E, I, R (disjoint masks of one
// 32-replica word of `node`): replica r moves iff its bit-sliced uniform is
// below its state's threshold.  All 32 replicas are compared at once; the
// first 8 planes decide all but 1 in 256 candidates, further planes are drawn
// only while some replica is undecided.  Returns the event mask.
//
// The 8-plane comparison runs from the least significant plane up, with one
// majority per plane: `less` keeps its value where uniform and threshold bits
// agree and becomes the threshold's bit where they differ, which is
// maj(~u, less, t).  The thresholds' bits come as masks from the constant bank
// (FlowThresholds); taken bit by bit from the 64-bit thresholds they cost more
// instructions than the two Philox calls.
__device__ __forceinline__ uint32_t maj_not(uint32_t u, uint32_t less, uint32_t t) {
  return (~u & (less | t)) | (less & t);
}
// Replicas whose threshold is 1 (they move without a draw).
__device__ __forceinline__ uint32_t flow_sure(uint32_t E, uint32_t I, uint32_t R,
                                              const FlowThresholds &th) {
  return (th.te_all ? E : 0u) | (th.ti_all ? I : 0u) | (th.tr_all ? R : 0u);
}
// The first th.lead planes (4, or 8) where every threshold has zeros: the
// replicas of `cand` whose uniform has them, too; the others do not move.
__device__ __forceinline__ uint32_t flow_top(uint32_t cand, const FlowThresholds &th,
                                             const uint32_t *rk, uint32_t node, uint32_t step,
                                             uint32_t word) {
  uint32_t x[8];
  if (th.lead >= 8) {
    philox4x32_10_rk_x2(node, step, word, 0u, 1u << 4, rk, x, x + 4);
    cand &= ~(x[4] | x[5] | x[6] | x[7]);
  } else {
    philox4x32_10_rk(node, step, word, 0u, rk, x);
  }
  return cand & ~(x[0] | x[1] | x[2] | x[3]);
}
// Events among the candidates `cand` (those flow_top left, with th.lead > 0).
__device__ __forceinline__ uint32_t flow_rest(uint32_t cand, uint32_t E, uint32_t I, uint32_t R,
                                              const FlowThresholds &th, const uint32_t *rk,
                                              uint32_t node, uint32_t step, uint32_t word) {
  const uint32_t e2 = E & cand, i2 = I & cand, r2 = R & cand;
  uint32_t x[4], less = 0, same = cand;
  if (th.lead < 8) {
    philox4x32_10_rk(node, step, word, 1u << 4, rk, x);
#pragma unroll
    for (int k = 7; k >= 4; --k) {
      const uint32_t t = (e2 & th.me[k]) | (i2 & th.mi[k]) | (r2 & th.mr[k]);
      less = maj_not(x[k - 4], less, t);
      same &= ~(t ^ x[k - 4]);
    }
  }
  if (th.lead < 4) {
    philox4x32_10_rk(node, step, word, 0u, rk, x);
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      const uint32_t t = (e2 & th.me[k]) | (i2 & th.mi[k]) | (r2 & th.mr[k]);
      less = maj_not(x[k], less, t);
      same &= ~(t ^ x[k]);
    }
  }
  uint32_t lt = less & cand;
#pragma unroll 1
  for (int j = 2; j < 16 && same != 0u; ++j) {
    philox4x32_10_rk(node, step, word, (uint32_t)j << 4, rk, x);
    const int sh = 60 - 4 * j;
    const uint32_t ce = (uint32_t)(th.te >> sh), ci = (uint32_t)(th.ti >> sh),
                   cr = (uint32_t)(th.tr >> sh);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t t = (((ce >> (3 - q)) & 1u) ? e2 : 0u) | (((ci >> (3 - q)) & 1u) ? i2 : 0u) |
                         (((cr >> (3 - q)) & 1u) ? r2 : 0u);
      lt |= same & t & ~x[q];
      same &= ~(t ^ x[q]);
    }
  }
  return lt;
}
// Candidates of a word: those whose threshold is neither 0 nor 1.
__device__ __forceinline__ uint32_t flow_candidates(uint32_t E, uint32_t I, uint32_t R,
                                                    const FlowThresholds &th) {
  return (th.te == 0 ? 0u : E) | (th.ti == 0 ? 0u : I) | (th.tr == 0 ? 0u : R);
}
__device__ __forceinline__ uint32_t flow_events(uint32_t E, uint32_t I, uint32_t R,
                                                const FlowThresholds &th, const uint32_t *rk,
                                                uint32_t node, uint32_t step, uint32_t word) {
  uint32_t cand = flow_candidates(E, I, R, th);
  const uint32_t sure = flow_sure(E, I, R, th);
  if (cand && th.lead) cand = flow_top(cand, th, rk, node, step, word);
  return cand ? sure | flow_rest(cand, E, I, R, th, rk, node, step, word) : sure;
}

// floor(p 2^64) for 0 < p < 1 (exact: p 2^64 is exact in float, then
// truncated).
__device__ __forceinline__ unsigned long long fixed64(float p) {
  return __float2ull_rz(__fmul_rn(p, 0x1p64f));
}

// Its top 8 bits (exact: p 2^8 is exact in float; one conversion to 32 bits
// instead of one to 64).
__device__ __forceinline__ uint32_t fixed8(float p) {
  return __float2uint_rz(__fmul_rn(p, 256.0f));
}

// Geometric infection uniform U_r of replica r, 64 bits, compared with
// floor(P 2^64).  Its top 8 bits are bit-sliced: bit k (k = 0 is 2^-1) is bit
// r % 32 of output k % 4 of counter (node, step, r / 32, 4 | (k / 4) << 4),
// so that two calls screen all 32 replicas of a word at once.  Its low 56
// bits are the top 56 bits of outputs 0-1 (output 0 high) of counter
// (node, step, r, 12), drawn only when the top 8 bits tie with the
// threshold's.
constexpr uint32_t kTagInfect = 4u;
constexpr uint32_t kTagInfectTail = 12u;

// The 8 planes of a word's infection uniforms.
__device__ __forceinline__ void infect_planes(const uint32_t *rk, uint32_t node, uint32_t step,
                                              uint32_t word, uint32_t pl[8]) {
  philox4x32_10_rk_x2(node, step, word, kTagInfect, kTagInfect | 16u, rk, pl, pl + 4);
}

// Top 8 bits of the uniform of replica bit b from its word's planes.
__device__ __forceinline__ uint32_t top8_of(const uint32_t pl[8], uint32_t b) {
  uint32_t u = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) u = __funnelshift_l(pl[k] << (31u - b), u, 1);
  return u;
}

// Replicas of `cand` whose top 8 uniform bits are at most t8 (< 256): with t8
// the top byte of a threshold, a superset of those below it.
__device__ __forceinline__ uint32_t top8_le(uint32_t cand, uint32_t t8, const uint32_t pl[8]) {
  // bits 7..4 and 3..0 of t8 as the sign bits of four bytes each, from which
  // one byte permute makes a mask
  const uint32_t hi = t8 * 0x08040201u, lo = (t8 << 4) * 0x08040201u;
  uint32_t le = 0xFFFFFFFFu;  // equal bits below: at most
#pragma unroll
  for (int k = 7; k >= 0; --k) {
    uint32_t t;  // the byte's sign, replicated
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(t) : "r"(k < 4 ? hi : lo), "r"(0x8888 + 0x1111 * (k & 3)));
    le = maj_not(pl[k], le, t);
  }
  return cand & le;
}

// Low 56 bits of the infection uniform of (global) replica `replica`.
__device__ __forceinline__ unsigned long long infect_tail56(const uint32_t *rk, uint32_t node,
                                                            uint32_t step, uint32_t replica) {
  uint32_t x[4];
  philox4x32_10_rk(node, step, replica, kTagInfectTail, rk, x);
  return (((unsigned long long)x[0] << 32) | x[1]) >> 8;
}

// Infection event of a replica whose uniform's top 8 bits are u8: event iff
// U < floor(P 2^64); P >= 1 always, P <= 0 or NaN never.
__device__ __forceinline__ bool infect_event(float P, uint32_t u8, const uint32_t *rk,
                                             uint32_t node, uint32_t step, uint32_t replica) {
  if (!(P > 0.0f)) return false;
  if (P >= 1.0f) return true;
  const uint32_t t8 = fixed8(P);
  if (u8 != t8) return u8 < t8;
  return infect_tail56(rk, node, step, replica) < (fixed64(P) & 0x00FFFFFFFFFFFFFFull);
}

// Countdown arithmetic of the reference (int op float, truncated back to
// int): c = (int)((float)c - step) and c = (int)((float)base + step).
__device__ __forceinline__ int32_t cd_sub(int32_t c, float step) {
  return __float2int_rz(__fsub_rn(__int2float_rn(c), step));
}
__device__ __forceinline__ int32_t cd_add(int32_t base, float step) {
  return __float2int_rz(__fadd_rn(__int2float_rn(base), step));
}

// Summary classification of a countdown value
// (tool/gpu_cpu_temporal_sim.cu:530-550): 0 S, 1 E, 2 I, 3 R.
__device__ __forceinline__ int countdown_class(int32_t c, int32_t E, int32_t I,
                                               int32_t R) {
  const int32_t upper = E + I + R;
  const int32_t elapsed = (c <= 0 || c > upper) ? 0 : (upper - c);
  if (c == 0) return 0;
  if (E > 0 && elapsed < E) return 1;
  if (I > 0 && elapsed < E + I) return 2;
  if (R > 0 && elapsed < E + I + R) return 3;
  return 0;
}

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

}  // namespace rp
