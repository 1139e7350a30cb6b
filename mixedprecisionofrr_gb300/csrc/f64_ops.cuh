// Short FP64 reciprocal, quotient and square root for latency-bound chains.
//
// An FP64 instruction takes this part's pipe 64 cycles, whatever it computes, so a division (~560 cycles) or square root
// (~630) is mostly its own refinement steps.  Here the reciprocal (or reciprocal root) of the 53-bit significand is
// formed to about 45 bits with FP32 pairs and integer operations alone, which run beside the FP64 pipe at full rate, and
// only the last step is FP64: Newton's for the reciprocal (two instructions), the exact-residual correction for
// quotient and root (three) [P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor,
// IBM J. Res. Dev. 34 (1990)].  Before its rounding a result is within 2^-86 of the exact one, so it is the correctly
// rounded value unless that lies within 2^-86 of a rounding boundary.  Whole families of operands do: divisors just
// below a power of two (1 / (2 - j 2^-52) is a boundary plus j^2 2^-107), and roots of operands beside a power of four.
// These, operands outside a wide exponent range, and zero, subnormal, infinite and NaN ones take the plain operation;
// roots of 1 + d for d < 2^-36, which a converging rotation asks for, the series 1 + (d / 2 - d^2 / 8).
// About 240, 310 and 310 cycles.
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

__device__ __forceinline__ double rcp(double x) {
  if (plain(x) || below_pow2(x)) return __drcp_rn(x);
  const double y = rcp_seed(x);
  return __fma_rn(y, __fma_rn(-y, x, 1.0), y);
}
__device__ __forceinline__ double div(double a, double b) {
  if (plain(a) || plain(b) || below_pow2(b) || (unsigned)(expo(a) - expo(b) + 800) > 1600u) return __ddiv_rn(a, b);
  const double y = rcp_seed(b), q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}
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
  return __fma_rn(__fma_rn(-g, g, x), hy, g);
}

}  // namespace f64
}  // namespace ofrr
