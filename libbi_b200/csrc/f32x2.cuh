// Packed FP32 arithmetic (fma/add/sub/mul.rn.f32x2) and Box-Muller in it.
//
// A packed instruction does two FP32 operations in one issue slot, at the
// same rate of the FP32 pipe (measured on B200: 3.3-3.9 warp operations per
// cycle and SM, scalar 3.8-3.9).  It pays where the issue slots are the
// limit: the four normals of a Philox block are two independent Box-Muller
// pairs, and side by side they take two thirds of the instructions (with the
// quotient and the square root below, which need no slow-path branch, a
// third less again).  Lorenz-96, d = 40, per step: 1000 particles 21.4 ->
// 17.4 us, 65536 particles 31.4 -> 30.1 us, the 256-filter batch's
// transition 643 -> 597 us, the guided step of 64 x 4096 178 -> 159 us.
// (RK4 itself in packed form, two particles per thread under 255 registers,
// was 5% faster still in the large batch, but slower everywhere else: it is
// bound by the FP32 pipe either way, and two warps per sub-partition hide
// little.)
//
// Every operation is rounded as the scalar one is, so the normals are the
// same bits as bpf_normal_pair_f's.  The assembler fuses a packed product
// into a packed sum: where a product must be rounded before it is added, one
// of the two stays scalar.
#pragma once
#include <stdint.h>
#include "../../include/bpf_math.h"

namespace bpf {
namespace pair {

typedef unsigned long long f2;  // two FP32 values

__device__ __forceinline__ f2 pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack(f2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 both(float a) { return pack(a, a); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 neg2(f2 a) { return a ^ 0x8000000080000000ull; }

// Two of bpf_normal_pair_f's pairs at once, from words (aA, bA) and (aB, bB):
// z0, z1 hold the first pair's normals in their low halves.  The
// quotient (m - 1)/(m + 1) and the square root are formed from the hardware's
// approximations with Markstein's corrections (P. W. Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J.
// Res. Dev. 34(1), 1990): one Newton step on the reciprocal, then q + r (n -
// q d); g + g'/2 (a - g g).  Over all 2^23 values of the uniform both equal
// the correctly rounded results.
__device__ __forceinline__ void normal_pair(uint32_t aA, uint32_t bA, uint32_t aB, uint32_t bB, f2& z0, f2& z1) {
  const f2 one = both(1.0f);
  // log u = log m + e ln 2, m in [sqrt(1/2), sqrt(2)) (bpf_logf_normal)
  const uint32_t uA = bpf_fbits(bpf_u01f(aA)), uB = bpf_fbits(bpf_u01f(aB));
  int eA = (int)(uA >> 23) - 127, eB = (int)(uB >> 23) - 127;
  float mA = bpf_bitsf((uA & 0x007FFFFFu) | 0x3F800000u), mB = bpf_bitsf((uB & 0x007FFFFFu) | 0x3F800000u);
  if (mA > 1.41421354f) { mA = mA * 0.5f; eA += 1; }
  if (mB > 1.41421354f) { mB = mB * 0.5f; eB += 1; }
  const f2 m = pack(mA, mB);
  const f2 num = sub2(m, one), den = add2(m, one), nden = neg2(den);
  float a, b;
  unpack(den, a, b);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(a));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(b));
  f2 r = pack(a, b);
  r = fma2(fma2(nden, r, one), r, r);
  const f2 q = mul2(num, r);
  const f2 s = fma2(fma2(nden, q, num), r, q);
  const f2 s2 = mul2(s, s);
  f2 p = fma2(both(1.0f / 9.0f), s2, both(1.0f / 7.0f));
  p = fma2(p, s2, both(1.0f / 5.0f));
  p = fma2(p, s2, both(1.0f / 3.0f));
  p = mul2(p, s2);
  const f2 t = add2(s, s);
  const f2 lm = fma2(t, p, t);
  const f2 ef = pack(bpf_small_int_to_float(eA), bpf_small_int_to_float(eB));
  const f2 lg = fma2(ef, both(0.693145751953125f), fma2(ef, both(1.428606765330187e-06f), lm));
  // the radius sqrt(-2 log u)
  const f2 w = mul2(both(-2.0f), lg);
  unpack(w, a, b);
  asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(a));
  asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(b));
  const f2 y = pack(a, b);
  const f2 g = mul2(w, y);
  const f2 rad = fma2(fma2(neg2(g), g, w), mul2(both(0.5f), y), g);
  // sin and cos of pi x, x = 2 u_b (bpf_sincospif_small)
  f2 x = pack(bpf_u01f(bA), bpf_u01f(bB));
  x = add2(x, x);
  const f2 tq = fma2(both(2.0f), x, both(12582912.0f));  // 2 x is exact
  const f2 qf = sub2(tq, both(12582912.0f));
  const f2 d = fma2(both(-0.5f), qf, x);
  const f2 d2 = mul2(d, d);
  f2 sn = fma2(both(0.08214588463306427f), d2, both(-0.5992645025253296f));
  sn = fma2(sn, d2, both(2.550163984298706f));
  sn = fma2(sn, d2, both(-5.167712688446045f));
  sn = fma2(sn, d2, both(3.1415927410125732f));
  sn = mul2(sn, d);
  f2 cs = fma2(both(-0.025806890800595284f), d2, both(0.23533062636852264f));
  cs = fma2(cs, d2, both(-1.3352627754211426f));
  cs = fma2(cs, d2, both(4.058712005615234f));
  cs = fma2(cs, d2, both(-4.934802055358887f));
  cs = fma2(cs, d2, one);
  // the quadrant: odd ones swap, the sine is negative in 2 and 3, the cosine
  // in 1 and 2
  float sA, sB, cA, cB, qA, qB;
  unpack(sn, sA, sB);
  unpack(cs, cA, cB);
  unpack(tq, qA, qB);
  const uint32_t iA = bpf_fbits(qA), iB = bpf_fbits(qB);
  const float s0 = (iA & 1u) ? cA : sA, c0 = (iA & 1u) ? sA : cA;
  const float s1 = (iB & 1u) ? cB : sB, c1 = (iB & 1u) ? sB : cB;
  z0 = mul2(rad, pack(bpf_bitsf(bpf_fbits(c0) ^ (((iA + 1u) & 2u) << 30)),
                      bpf_bitsf(bpf_fbits(c1) ^ (((iB + 1u) & 2u) << 30))));
  z1 = mul2(rad, pack(bpf_bitsf(bpf_fbits(s0) ^ ((iA & 2u) << 30)), bpf_bitsf(bpf_fbits(s1) ^ ((iB & 2u) << 30))));
}

}  // namespace pair
}  // namespace bpf
