// Square roots and reciprocals in few FP64 instructions.
#pragma once

#include <cuda_runtime.h>

namespace ptn {

// 1 / sqrt(d) and 1 / d from an FP32 seed y and one step of third order (Householder's
// iteration): with the defect r = 1 - d y^2 (or 1 - d y) of the seed, |r| < 2^-21,
//   1 / sqrt(d) = y (1 - r)^(-1/2) = y (1 + r / 2 + 3 r^2 / 8 + ...),
//   1 / d = y (1 - r)^(-1) = y (1 + r + r^2 + ...),
// the series cut where the next term is below 2^-63. Seed and scaling are integer work on the
// IEEE fields: five and three FP64 instructions (64 cycles each on this part) where the division
// and square root sequences take several times that. Within 2^-52 of the exact value;
// subnormal, zero and non-finite arguments take the CUDA functions.
__device__ __forceinline__ double seed_scale(float y, int e) {   // y 2^e for a normal float y
  const unsigned b = __float_as_uint(y);
  const int x = (int)(b >> 23) - 127 + 1023 + e;
  return __longlong_as_double(((long long)x << 52) | ((long long)(b & 0x7FFFFFu) << 29));
}

// 1 / sqrt(x^2 + y^2), the same way, for sums near 1 .. 2
__device__ __forceinline__ double inv_norm(double x, double y) {
  const double d = fma(x, x, y * y);
  const double s = (double)rsqrtf((float)d);
  const double e = fma(-d * s, s, 1.0);
  return fma(s * e, fma(e, 0.375, 0.5), s);
}

// y / 2 of a normal y well above the subnormal range, without an FP64 instruction
__device__ __forceinline__ double half_of(double y) {
  return __longlong_as_double(__double_as_longlong(y) - (1LL << 52));
}

__device__ __forceinline__ double fast_rsqrt(double d) {
  const long long b = __double_as_longlong(d);
  const int E = (int)((b >> 52) & 0x7FF);
  if (b <= 0 || E == 0 || E == 0x7FF) return 1.0 / sqrt(d);
  const int e = E - 1023, odd = e & 1;
  const float m = __uint_as_float(((unsigned)(127 + odd) << 23) | ((unsigned)(b >> 29) & 0x7FFFFFu));
  const double y = seed_scale(rsqrtf(m), -(e - odd) / 2);
  const double r = fma(-(d * y), y, 1.0);
  return fma(y * r, fma(r, 0.375, 0.5), y);
}

__device__ __forceinline__ double fast_recip(double d) {   // d > 0
  const long long b = __double_as_longlong(d);
  const int E = (int)((b >> 52) & 0x7FF);
  if (b <= 0 || E < 2 || E > 2040) return 1.0 / d;
  const float m = __uint_as_float(0x3F800000u | ((unsigned)(b >> 29) & 0x7FFFFFu));
  const double y = seed_scale(__frcp_rn(m), -(E - 1023));
  const double r = fma(-d, y, 1.0);
  return fma(y, fma(r, r, r), y);
}

}  // namespace ptn
