// Sine and cosine together, in fp32, for the feature maps that keep fp32's precision.
//
// Cody and Waite's reduction by pi / 2 in three fp32 parts (each step one rounding), then minimax polynomials on [-pi / 4, pi / 4] (odd
// and even, three coefficients each, fitted by Lawson's iteration: 3.6e-9 relative and 9.6e-11 absolute in front of fp32's rounding).
// At most 1.6 units in the last place, 2.1e-8 in the mean square, up to |x| = 8000; beyond, and for NaN, the library's.  22
// instructions a pair, where the library's function, with its reduction for all of fp32's range in line, takes about 75.
#pragma once

#include <cuda_runtime.h>

namespace rfa {

constexpr float kTrigMax = 8000.f;
static __device__ __noinline__ float2 sincos_large(float x) {
  float2 r;
  sincosf(x, &r.x, &r.y);
  return r;
}
__device__ __forceinline__ void fm_sincos(float x, float& s, float& c) {
  const float k0 = fmaf(x, 0.636619772f, 12582912.f), k = k0 - 12582912.f;
  const int q = __float_as_int(k0);
  const float r = fmaf(k, 1.7151245e-15f, fmaf(k, 4.37113883e-8f, fmaf(k, -1.57079637f, x))), z = r * r;
  const float sp = fmaf(z * r, fmaf(fmaf(-1.9516978e-4f, z, 8.3321761e-3f), z, -1.6666655e-1f), r);
  const float cp = fmaf(z * z, fmaf(fmaf(2.443809e-5f, z, -1.3887364e-3f), z, 4.1666646e-2f), fmaf(z, -0.5f, 1.f));
  s = __int_as_float(__float_as_int(q & 1 ? cp : sp) ^ ((q & 2) << 30));
  c = __int_as_float(__float_as_int(q & 1 ? sp : cp) ^ (((q + 1) & 2) << 30));
  if (!(fabsf(x) <= kTrigMax)) {
    const float2 l = sincos_large(x);
    s = l.x; c = l.y;
  }
}

}  // namespace rfa
