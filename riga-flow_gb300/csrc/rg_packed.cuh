// rg_packed.cuh — packed FP32x2 forms (sm_100 and later) of the FP32 lanes' functions.
#pragma once
#include "rg_common.cuh"

// rg_probit32 of two points in packed FP32x2 arithmetic, each with rg_probit32's operations.
__device__ __forceinline__ float2 rg_probit32x2(uint32_t xa, uint32_t xb) {
  auto both = [](float a) { return make_float2(a, a); };
  const uint32_t ya = xa ^ (uint32_t)((int32_t)xa >> 31), yb = xb ^ (uint32_t)((int32_t)xb >> 31);  // min(x, ~x)
  const float2 c = both(4.656612873077393e-10f), h = both(2.3283064365386963e-10f);
  const float2 p2 = __ffma2_rn(make_float2((float)(int32_t)ya, (float)(int32_t)yb), c, h);
  const float2 s = __ffma2_rn(make_float2((float)(int32_t)(ya ^ 0x7FFFFFFFu), (float)(int32_t)(yb ^ 0x7FFFFFFFu)), c, h);
  const float2 v = __ffma2_rn(p2, s, p2);
  const float2 w = make_float2(rg_neg_ln(v.x), rg_neg_ln(v.y));
  const float2 t = __fadd2_rn(w, both(-2.5f));
  float2 g = both(4.035466097e-08f);
  g = __ffma2_rn(g, t, both(4.861039695e-07f));
  g = __ffma2_rn(g, t, both(-4.990565522e-06f));
  g = __ffma2_rn(g, t, both(-6.217993119e-06f));
  g = __ffma2_rn(g, t, both(3.091502040e-04f));
  g = __ffma2_rn(g, t, both(-1.773010155e-03f));
  g = __ffma2_rn(g, t, both(-5.908170971e-03f));
  g = __ffma2_rn(g, t, both(3.488026599e-01f));
  g = __ffma2_rn(g, t, both(2.123313567e+00f));
  if (fmaxf(w.x, w.y) >= 5.0f) {  // 0.7% of pairs
    if (w.x >= 5.0f) g.x = rg_ninv32_tail(w.x);
    if (w.y >= 5.0f) g.y = rg_ninv32_tail(w.y);
  }
  const float2 q = __fmul2_rn(s, g);
  // negative in the lower half
  return make_float2(__uint_as_float(__float_as_uint(q.x) ^ (~xa & 0x80000000u)),
                     __uint_as_float(__float_as_uint(q.y) ^ (~xb & 0x80000000u)));
}
