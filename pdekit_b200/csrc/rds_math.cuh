// Reciprocal and reciprocal square root in FP64 without branches, for chains that the compiler
// should overlap between nodes or points: the library division and rsqrt branch on special
// values, which keeps independent evaluations of an unrolled loop apart.
//
// Both start from the PTX approximations (relative error below 2^-19) and take one step of a
// third-order iteration, so the error left is that of its own roundings (about one unit in the
// last place; tests/cpp/math_test.cu). With e = 1 - x y the reciprocal is y / (1 - e), expanded
// to y (1 + e + e^2); with e = 1 - x y^2 the reciprocal square root is y (1 - e)^(-1/2), expanded
// to y (1 + e / 2 + 3 e^2 / 8) (Householder's iterations of order three).
#pragma once

#include <cuda_runtime.h>

namespace rds
{

// 1 / x for finite normal x; NaN where 1 / x is infinite, 0 or denormal.
__device__ __forceinline__ double rcp_fast(double x)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(fma(e, e, e), y, y);
}

// 1 / sqrt(x) for finite normal x > 0; NaN for other x.
__device__ __forceinline__ double rsqrt_fast(double x)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  return fma(fma(e, 0.375, 0.5), y * e, y);
}

__device__ __forceinline__ float rcp_fast(float x) { return 1.f / x; }

// sqrt(x) for x > 0, and the reciprocal of the result in FP64. FP32: the correctly rounded root
// (x rsqrtf(x) is off by up to 2 units in the last place).
__device__ __forceinline__ double sqrt_and_inverse(double x, double &inv)
{
  inv = rsqrt_fast(x);
  return x * inv;
}
__device__ __forceinline__ float sqrt_and_inverse(float x, double &inv)
{
  const float s = sqrtf(x);
  inv           = rcp_fast(double(s));
  return s;
}

// max(0, x), and x < y of numbers that are not negative. FP64: integer tests, since a comparison
// would take a slot of the FP64 pipe, which bounds these kernels.
__device__ __forceinline__ double pos_part(double x) { return __double2hiint(x) < 0 ? 0.0 : x; }
__device__ __forceinline__ float pos_part(float x) { return x > 0.f ? x : 0.f; }
__device__ __forceinline__ bool less_pos(double x, double y)
{
  return __double_as_longlong(x) < __double_as_longlong(y);
}
__device__ __forceinline__ bool less_pos(float x, float y) { return x < y; }

// x y, rounded (not fused into a sum that uses it).
__device__ __forceinline__ double mul_rn(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ float mul_rn(float x, float y) { return __fmul_rn(x, y); }

} // namespace rds
