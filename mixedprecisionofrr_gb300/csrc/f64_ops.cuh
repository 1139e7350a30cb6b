// Short FP64 reciprocal, quotient and square root for latency-bound chains: the correctly rounded values.
//
// An FP64 instruction takes this part's pipe 64 cycles, whatever it computes, so a division (~565 cycles) or square root
// (~600) is mostly its own refinement steps.  Here the reciprocal (or reciprocal root) of the 53-bit significand is
// formed to about 45 bits with FP32 pairs and integer operations alone, which run beside the FP64 pipe at full rate, and
// only the last step is FP64: Newton's for the reciprocal (two instructions), the residual correction for
// quotient and root (three) [P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor,
// IBM J. Res. Dev. 34 (1990)].  Before its rounding a result is within 2^-86 of the exact one, so it is the correctly
// rounded value or its neighbour: exact values come as close as 2^-107 to a rounding boundary (1.5 / (1 + 2^-52), or any
// a 2^54 = b m + r with m odd and r small; one random operand in 2^33).  The remainder, formed exactly in 64-bit integers
// (it is below 2^55, so the low words of the products suffice), decides between the two; no quotient or root lies on a
// boundary itself.  Without that decision (RN = false) the error is below 1/2 + 2^-33 units in the last place.
// Operands outside a wide exponent range, and zero, subnormal, infinite and NaN ones take the plain operation; so do
// divisors and radicands just below a power of two (the seed's binade, and the root's, change there); roots of 1 + d for
// d < 2^-36, which a converging rotation asks for, the series 1 + (d / 2 - d^2 / 8).
// In a lone warp, cycles: reciprocal 310, quotient 400, root 455 (240, 325 and 380 with RN = false) against 350, 565 and
// 600 of the plain operations.
#pragma once
#include <cuda_runtime.h>

namespace ofrr {
namespace f64 {

__device__ __forceinline__ int expo(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ bool plain(double x) { return (unsigned)(expo(x) - 200) > 1646u; }  // exponent field 200..1846
__device__ __forceinline__ bool below_pow2(double x) { return (__double2hiint(x) & 0xfffff) == 0xfffff; }

// the significand of x in [1, 2) as FP32 pair (46 bits), the upper part at least
__device__ __forceinline__ void split(double x, float* h, float* l) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  *h = __uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29));
  *l = (__uint_as_float(0x4b000000u | ((lo >> 6) & 0x7fffffu)) - 8388608.f) * 1.4210854715202004e-14f;  // 2^-46
}
// y0 + y1 (y0 in (1/2, 1), |y1| < 2^-20) as the significand part of a double with exponent field `field` for [1/2, 1)
__device__ __forceinline__ double join(float y0, float y1, int field, unsigned sign) {
  const unsigned b0 = __float_as_uint(y0);
  long long m = ((long long)(b0 & 0x7fffffu) << 29) + ((long long)__float2int_rn(y1 * 1125899906842624.f) << 3);  // 2^50
  m += (long long)field << 52;
  return __longlong_as_double(m | ((long long)sign << 32));
}

// 1 / x to about 45 bits (plain(x) false)
__device__ __forceinline__ double rcp_seed(double x) {
  float h, l, y0;
  split(x, &h, &l);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(h));
  y0 = fminf(y0, 0.99999994f);  // inside (1/2, 1)
  float r = fmaf(-h, y0, 1.f);  // exact
  r = fmaf(-l, y0, r);
  return join(y0, y0 * fmaf(r, r, r), 2045 - expo(x), (unsigned)__double2hiint(x) & 0x80000000u);
}
// 1 / sqrt(x) to about 45 bits (x > 0, plain(x) false)
__device__ __forceinline__ double rsqrt_seed(double x) {
  float h, l, y0;
  split(x, &h, &l);
  const int e = expo(x) - 1023;
  const bool odd = e & 1;
  if (odd) {  // significand in [2, 4)
    h *= 2.f;
    l *= 2.f;
  }
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(h));
  y0 = fminf(fmaxf(y0, 0.50000006f), 0.99999994f);
  const float p = y0 * y0, pe = fmaf(y0, y0, -p);
  float r = fmaf(-h, p, 1.f);
  r = fmaf(-h, pe, r);
  r = fmaf(-l, p, r);
  return join(y0, y0 * (r * fmaf(0.375f, r, 0.5f)), 1022 - ((e - (odd ? 1 : 0)) >> 1), 0u);
}

// the significand as an integer in [2^52, 2^53)
__device__ __forceinline__ unsigned long long sig(double x) {
  return ((unsigned long long)__double_as_longlong(x) & 0xfffffffffffffull) | (1ull << 52);
}
// the low 64 bits of s 2^k, 32 <= k < 64
__device__ __forceinline__ unsigned long long shl_low(unsigned long long s, int k) {
  return (unsigned long long)((unsigned)s << (k - 32)) << 32;
}
// x for 0 <= u <= top; else its neighbour nearer zero (u < 0) or further from it
__device__ __forceinline__ double settle(double x, unsigned long long u, unsigned long long top) {
  const int n = (int)((long long)u >> 63) | 1;  // -1 or 1
  return __longlong_as_double(__double_as_longlong(x) + (u > top ? n : 0));
}

template <bool RN = true>
__device__ __forceinline__ double rcp(double x) {
  if (plain(x) || below_pow2(x)) return __drcp_rn(x);
  const double s = rcp_seed(x), y = __fma_rn(s, __fma_rn(-s, x, 1.0), s);
  if (!RN) return y;
  // the remainder 2^104 (or 2^105) - X Y in [-X / 2, X / 2]
  const unsigned long long X = sig(x);
  return settle(y, X + (0ull - 2 * X) * sig(y), 2 * X);
}
template <bool RN = true>
__device__ __forceinline__ double div(double a, double b) {
  if (plain(a) || plain(b) || below_pow2(b) || (unsigned)(expo(a) - expo(b) + 800) > 1600u) return __ddiv_rn(a, b);
  const double y = rcp_seed(b), q0 = __dmul_rn(a, y), q = __fma_rn(__fma_rn(-b, q0, a), y, q0);
  if (!RN) return q;
  // the remainder A 2^k - B Q in [-B / 2, B / 2]; Q has 53 bits with k = 52 for A >= B, else with k = 53
  const unsigned long long A = sig(a), B = sig(b);
  return settle(q, (shl_low(A, A < B ? 54 : 53) + B) + (0ull - 2 * B) * sig(q), 2 * B);
}
template <bool RN = true>
__device__ __forceinline__ double sqrt(double x) {
  if (plain(x) || below_pow2(x) || __double2hiint(x) < 0) return __dsqrt_rn(x);
  if ((__double2hiint(x) & 0x1fffff) == 0x100000 && (unsigned)__double2loint(x) < 65536u) {  // 4^k (1 + d), d < 2^-36
    const int k = (expo(x) - 1023) >> 1;
    const double d = __dadd_rn(__hiloint2double(0x3ff00000, __double2loint(x)), -1.0);  // exact
    const double c = __fma_rn(__dmul_rn(d, d), -0.125, __dmul_rn(0.5, d)), s1 = __dadd_rn(1.0, c);
    return __hiloint2double(__double2hiint(s1) + k * (1 << 20), __double2loint(s1));
  }
  const double y = rsqrt_seed(x), g = __dmul_rn(x, y);
  const double hy = __hiloint2double(__double2hiint(y) - (1 << 20), __double2loint(y));  // y / 2
  const double r = __fma_rn(__fma_rn(-g, g, x), hy, g);
  if (!RN) return r;
  // the remainder X 2^k - G^2 (k = 52, or 53 for an odd exponent) in [1 - G, G], as (G +- 1/2)^2 - G^2 = +-G + 1/4
  const unsigned long long G = sig(r), K = shl_low(sig(x), 53 - (expo(x) & 1)) - 1;
  return settle(r, K + (1 - G) * G, 2 * G - 1);
}

}  // namespace f64
}  // namespace ofrr
