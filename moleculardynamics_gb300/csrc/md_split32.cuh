// Differences of FP64 coordinates to FP32 without FP64 operations (conversions and
// differences there take GB300's narrow FP64 pipe): a coordinate is the sum of two
// FP32 numbers.  Compiled for the host as well.
#pragma once
#include "md_exact64.cuh"

namespace mdgb {

// x as the sum of two FP32 numbers, by moving the fields: 24 and 24 bits of the 53
__host__ __device__ __forceinline__ float2 split64(double x) {
#ifdef __CUDA_ARCH__
  const uint64_t b = (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  __builtin_memcpy(&b, &x, 8);
#endif
  const uint32_t e = (uint32_t)(b >> 52) & 0x7FFu;
  // the low 29 bits of the mantissa, worth 2^(e - 1075) each
  const uint32_t ub = e > 948u && e < 1151u ? (e - 948u) << 23 : 0u;
#ifdef __CUDA_ARCH__
  const float u = __uint_as_float(ub);
#else
  float u;
  __builtin_memcpy(&u, &ub, 4);
#endif
  const float l = (float)((uint32_t)b & 0x1FFFFFFFu) * u;
  return make_float2(trunc32(x), b >> 63 ? -l : l);
}

// s + e = a + b
__host__ __device__ __forceinline__ float two_sum(float a, float b, float& e) {
  const float s = a + b, t = s - a;
  e = (a - (s - t)) + (b - t);
  return s;
}

// x_j + img box - x_i, rounded once to FP32 but for the parts' own roundings (2^-47
// of the coordinates).  The upper parts' difference keeps its rounding error: where
// they differ in sign or size, as near the planes through the origin, dropping it
// made the result up to a unit in the last place off, not half a unit.
__host__ __device__ __forceinline__ float diff32(float2 xj, float2 xi, int img, float2 box) {
  float s = xj.x, l = xj.y - xi.y, e;
  if (img) {
    s = two_sum(xj.x, img > 0 ? box.x : -box.x, e);
    l += e + (img > 0 ? box.y : -box.y);
  }
  const float d = two_sum(s, -xi.x, e);
  return d + (e + l);
}

}  // namespace mdgb
