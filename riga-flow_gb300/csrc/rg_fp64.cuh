// rg_fp64.cuh — FP64 building blocks of the parity kernels with fewer operations on the FP64 pipe.
//
// GB300 issues about one FP64 warp instruction per 16 clocks and SM, 64 times fewer than its
// integer and FP32 instructions, so everything that is exact by construction leaves that pipe:
// comparisons of magnitudes, scalings by powers of two, conversions of small integers and range
// checks run on the bit patterns, and a division starts from an FP32 reciprocal.  Every function
// returns the bits of the one it stands in for (rg_exp64, rg_log64, rg_probit64, a / b), which
// round each product and sum separately.  Compiled without FMA contraction; the fused operations
// below are written out.
#pragma once
#include "rg_common.cuh"

namespace rg {

__device__ __forceinline__ int hi_word(double x) { return __double2hiint(x); }
// x·2^k for a normal x whose result is normal.
__device__ __forceinline__ double scale_pow2(double x, int k) {
  return __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x));
}
// x / 2, exact.
__device__ __forceinline__ double halve(double x) {
  const uint32_t e = (uint32_t)__double2hiint(x) & 0x7ff00000u;
  return e - 0x00200000u < 0x7fd00000u ? scale_pow2(x, -1) : 0.5 * x;  // zeros, subnormals, infinities, NaNs
}
// The integer as a double, by the bits of 1.5·2^52 + i.
__device__ __forceinline__ double small_int(int i) {
  return __longlong_as_double(0x4338000000000000LL + i) - 6755399441055744.0;
}
// Doubles in order as signed integers (NaNs beyond the infinities of their sign).
__device__ __forceinline__ long long order_key(double x) {
  const long long b = __double_as_longlong(x);
  return (b << 1) == 0 ? 0 : b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

// 1 / d within half an ulp and 2^-66 of itself for |d| in FP32's normal range: an FP32 reciprocal of d's
// leading bits (|e| below 2^-22 with the bits cut off) and one cubic step y(1 + e + e²), e = 1 - d·y.
__device__ __forceinline__ double reciprocal(double d) {
  const int h = __double2hiint(d);
  const uint32_t f = ((uint32_t)h & 0x80000000u) | ((((uint32_t)h & 0x7fffffffu) - (896u << 20)) << 3) |
                     ((uint32_t)__double2loint(d) >> 29);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  const uint32_t b = __float_as_uint(r);
  const double y = __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
  double e = __fma_rn(-d, y, 1.0);
  e = __fma_rn(e, e, e);
  return __fma_rn(y, e, y);
}
// n / d rounded to nearest, given y = 1 / d: the quotient estimate corrected by its exact remainder
// (Markstein, IBM J. Res. Dev. 34, 1990).  For normal n (or zero) and quotients.  With significands d in
// [1, 2) and quotients in [1, 2), the corrected value is off by |q - n/d|·d·|y - 1/d| before it is rounded,
// at most about 2^-107·d near a midpoint of two doubles, and an exact quotient stays 2^-105 / d or more away from
// every midpoint, so the result is correctly rounded for a rounded y, and for `reciprocal`'s unless d is
// within 2^-12 of 2.  There no case is known: the hardest quotients of the 2^22 divisors next below 2 and of
// 2^25 others all round correctly (tests/test_fp64_blocks_gpu.py).
__device__ __forceinline__ double divide_by(double n, double d, double y) {
  const double q = n * y;
  return __fma_rn(__fma_rn(-d, q, n), y, q);
}
// n / d for |d| in FP32's normal range and normal (or zero) n and quotient.
__device__ __forceinline__ double divide(double n, double d) { return divide_by(n, d, reciprocal(d)); }

// The general forms, kept out of line: merged into the fast ones they bring their range checks along
// (five FP64 comparisons a step).
__device__ __noinline__ static double general_exp64(double x) { return rg_exp64(x); }
__device__ __noinline__ static double general_log64(double x) { return rg_log64(x); }

// rg_exp64.  Below |x| = 0.34 its reduction is the identity (k = 0).
__device__ __forceinline__ double fast_exp64(double x) {
  if (((uint32_t)hi_word(x) & 0x7fffffffu) >= 0x3fd5c28fu) return general_exp64(x);
  double p = 0x1.6124613a86d09p-33;
  p = p * x + 0x1.1eed8eff8d898p-29;
  p = p * x + 0x1.ae64567f544e4p-26;
  p = p * x + 0x1.27e4fb7789f5cp-22;
  p = p * x + 0x1.71de3a556c734p-19;
  p = p * x + 0x1.a01a01a01a01ap-16;
  p = p * x + 0x1.a01a01a01a01ap-13;
  p = p * x + 0x1.6c16c16c16c17p-10;
  p = p * x + 0x1.1111111111111p-7;
  p = p * x + 0x1.5555555555555p-5;
  p = p * x + 0x1.5555555555555p-3;
  p = p * x + 0.5;
  p = p * x + 1.0;
  return p * x + 1.0;
}

// rg_log64 of a positive normal x.
__device__ __forceinline__ double fast_log64(double x) {
  const long long b = __double_as_longlong(x);
  int e = (int)(b >> 52) - 1023;
  long long mb = (b & 0x000fffffffffffffLL) | 0x3ff0000000000000LL;
  if (mb > 0x3ff6a09e667f3bcdLL) {  // the mantissa is above sqrt(2)
    mb -= 0x0010000000000000LL;
    ++e;
  }
  const double f = __longlong_as_double(mb) - 1.0;
  const double s = divide(f, 2.0 + f);
  const double z = s * s;
  double R = 0x1.642c8590b2164p-5;
  R = R * z + 0x1.8618618618618p-5;
  R = R * z + 0x1.af286bca1af28p-5;
  R = R * z + 0x1.e1e1e1e1e1e1ep-5;
  R = R * z + 0x1.1111111111111p-4;
  R = R * z + 0x1.3b13b13b13b14p-4;
  R = R * z + 0x1.745d1745d1746p-4;
  R = R * z + 0x1.c71c71c71c71cp-4;
  R = R * z + 0x1.2492492492492p-3;
  R = R * z + 0x1.999999999999ap-3;
  R = R * z + 0x1.5555555555555p-2;
  R = R * z;
  const double t = s + s * R;
  const double lm = mb == 0x3ff0000000000000LL ? 0.0 : scale_pow2(t, 1);  // f = 0, or |t| >= 2^-54
  const double ed = small_int(e);
  return ed * 0x1.62e42ffp-1 + (lm + ed * -0x1.718432a1b0e26p-35);
}

// rg_probit64 of u = (x + 1/2) / 2^32 (whose clamp to [1e-12, 1 - 1e-12] never acts).
__device__ __forceinline__ bool probit64_is_tail(uint32_t x) {
  // u < 0.02425 or u > 1 - 0.02425
  return x < 104152957u || x > 4190814338u;
}
__device__ __forceinline__ double probit64_central(uint32_t x) {
  // 2^51 + x + 1/2 by its bits, whose last place is 1/2; then x + 1/2 - 2^31 exactly, and q = u - 1/2
  const uint32_t m = 2u * x + 1u;
  const double d = __hiloint2double((int)(0x43200000u | (x >> 31)), (int)m) - 2251801961168896.0;
  const double q = scale_pow2(d, -32), r = q * q;
  const double num = (((((-3.969683028665376e1 * r + 2.209460984245205e2) * r + -2.759285104469687e2) * r +
                        1.383577518672690e2) * r + -3.066479806614716e1) * r + 2.506628277459239e0) * q;
  const double den = ((((-5.447609879822406e1 * r + 1.615858368580409e2) * r + -1.556989798598866e2) * r +
                       6.680131188771972e1) * r + -1.328068155288572e1) * r + 1.0;
  return divide(num, den);
}
__device__ __forceinline__ double probit64_tail(uint32_t x) {
  const bool low = x < 0x80000000u;
  // min(u, 1 - u), exact either way
  const double p = ((double)(low ? x : ~x) + 0.5) * 2.3283064365386962890625e-10;
  const double q = sqrt(-2.0 * fast_log64(p));
  const double v = (((((-7.784894002430293e-3 * q + -3.223964580411365e-1) * q + -2.400758277161838e0) * q +
                      -2.549732539343734e0) * q + 4.374664141464968e0) * q + 2.938163982698783e0) /
                   ((((7.784695709041462e-3 * q + 3.224671290700398e-1) * q + 2.445134137142996e0) * q +
                     3.754408661907416e0) * q + 1.0);
  return low ? v : -v;
}

}  // namespace rg
