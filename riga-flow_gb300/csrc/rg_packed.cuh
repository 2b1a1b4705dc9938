// rg_packed.cuh — packed FP32x2 forms (sm_100 and later) of the FP32 lanes' functions.
#pragma once
#include "rg_common.cuh"

// rg_ninv32_tail of two arguments.
__device__ __forceinline__ float2 rg_ninv32_tail2(float2 w) {
  auto both = [](float a) { return make_float2(a, a); };
  const float2 v = __fadd2_rn(make_float2(sqrtf(w.x), sqrtf(w.y)), both(-3.716110200f));
  float2 g = both(5.467908077e-06f);
  g = __ffma2_rn(g, v, both(-1.174909974e-05f));
  g = __ffma2_rn(g, v, both(-2.363354380e-05f));
  g = __ffma2_rn(g, v, both(9.947906459e-05f));
  g = __ffma2_rn(g, v, both(-1.555746239e-04f));
  g = __ffma2_rn(g, v, both(2.347132999e-04f));
  g = __ffma2_rn(g, v, both(-4.239792245e-04f));
  g = __ffma2_rn(g, v, both(8.495624679e-04f));
  g = __ffma2_rn(g, v, both(-1.928687814e-03f));
  g = __ffma2_rn(g, v, both(3.093904488e-03f));
  g = __ffma2_rn(g, v, both(1.426282266e+00f));
  g = __ffma2_rn(g, v, both(5.025157229e+00f));
  return g;
}
// rg_probit32 of K pairs of points in packed FP32x2 arithmetic, each with rg_probit32's operations.  The
// pairs go through the polynomial in step, so that each coefficient is brought into a register pair once
// for all of them, and through one test for the tail, which leaves one branch instead of K.  Against one
// pair at a time: the books' generation of 20 assets 61.9 -> 58.2 ms a book, a 3-asset quote of 2^13
// paths 203 -> 197 us, 2^21 paths of 5 assets on the direct kernel 35.6 -> 34.4 ms.
template <int K>
__device__ __forceinline__ void rg_probit32x2(const uint32_t (&xa)[K], const uint32_t (&xb)[K], float2 (&out)[K]) {
  auto both = [](float a) { return make_float2(a, a); };
  float2 s[K], t[K], g[K];  // the upper point's half, signed; the logarithm's distance to 2.5
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint32_t ya = xa[k] ^ (uint32_t)((int32_t)xa[k] >> 31), yb = xb[k] ^ (uint32_t)((int32_t)xb[k] >> 31);  // min(x, ~x)
    const float2 c = both(4.656612873077393e-10f), h = both(2.3283064365386963e-10f);
    const float2 p2 = __ffma2_rn(make_float2((float)(int32_t)ya, (float)(int32_t)yb), c, h);
    const float2 u = __ffma2_rn(make_float2((float)(int32_t)(ya ^ 0x7FFFFFFFu), (float)(int32_t)(yb ^ 0x7FFFFFFFu)), c, h);
    const float2 v = __ffma2_rn(p2, u, p2);
    // single products: a packed one is contracted with the sum into one rounding
    t[k] = __fadd2_rn(make_float2(rg_neg_ln(v.x), rg_neg_ln(v.y)), both(-2.5f));
    // negative in the lower half
    s[k] = make_float2(__uint_as_float(__float_as_uint(u.x) ^ (~xa[k] & 0x80000000u)),
                       __uint_as_float(__float_as_uint(u.y) ^ (~xb[k] & 0x80000000u)));
    g[k] = both(4.035466097e-08f);
  }
  constexpr float kG[8] = {4.861039695e-07f,  -4.990565522e-06f, -6.217993119e-06f, 3.091502040e-04f,
                           -1.773010155e-03f, -5.908170971e-03f, 3.488026599e-01f,  2.123313567e+00f};
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int k = 0; k < K; ++k) g[k] = __ffma2_rn(g[k], t[k], both(kG[i]));
  // w >= 5, 0.4% of points; w = t + 2.5 is exact there
  float far = fmaxf(t[0].x, t[0].y);
#pragma unroll
  for (int k = 1; k < K; ++k) far = rg_max3(far, t[k].x, t[k].y);
  if (far >= 2.5f) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (fmaxf(t[k].x, t[k].y) >= 2.5f) {
        const float2 far_g = rg_ninv32_tail2(__fadd2_rn(t[k], both(2.5f)));
        if (t[k].x >= 2.5f) g[k].x = far_g.x;
        if (t[k].y >= 2.5f) g[k].y = far_g.y;
      }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) out[k] = __fmul2_rn(s[k], g[k]);
}
