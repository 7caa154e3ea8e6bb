// 2^x of two lanes, as the softmax of the tensor-core forward kernels evaluates it.
#pragma once
#include "ar_ptx.cuh"

namespace ar {
using namespace arptx;

// 2^x for two lanes on the MUFU unit.
__device__ __forceinline__ void exp2_mufu_x2(uint64_t x2, float& p0, float& p1) {
  float a, b;
  unpack_f32x2(x2, a, b);
  p0 = ex2f(a);
  p1 = ex2f(b);
}
// 2^x for two lanes without the MUFU unit: x = n + f with n the nearest integer (read from the low mantissa bits of
// x + 1.5 * 2^23) and f in [-0.5, 0.5], 2^f by a cubic whose relative error stays below 1.1e-4 (P is rounded to
// bf16, 2^-9, afterwards), n added to the exponent field.  x is clamped at -126 so that the exponent cannot wrap;
// 2^0 is exactly 1.
__device__ __forceinline__ void exp2_poly_x2(uint64_t x2, float& p0, float& p1) {
  float a, b;
  unpack_f32x2(x2, a, b);
  const uint64_t xc = pack_f32x2(fmaxf(a, -126.0f), fmaxf(b, -126.0f));
  const uint64_t t2 = add_f32x2(xc, pack_f32x2(12582912.0f, 12582912.0f));
  const uint64_t n2 = add_f32x2(t2, pack_f32x2(-12582912.0f, -12582912.0f));
  const uint64_t f2 = fma_f32x2(n2, pack_f32x2(-1.0f, -1.0f), xc);
  uint64_t y2 = fma_f32x2(pack_f32x2(0.055008914f, 0.055008914f), f2, pack_f32x2(0.242211f, 0.242211f));
  y2 = fma_f32x2(y2, f2, pack_f32x2(0.69328296f, 0.69328296f));
  y2 = fma_f32x2(y2, f2, pack_f32x2(1.0f, 1.0f));
  float ya, yb, ta, tb;
  unpack_f32x2(y2, ya, yb);
  unpack_f32x2(t2, ta, tb);
  p0 = __uint_as_float(__float_as_uint(ya) + (__float_as_uint(ta) << 23));
  p1 = __uint_as_float(__float_as_uint(yb) + (__float_as_uint(tb) << 23));
}

}  // namespace ar
