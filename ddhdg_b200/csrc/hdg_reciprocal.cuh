// Reciprocals of pivots, shared by the eliminations (sm_100a).
//
// 1 / x by two Newton steps from the hardware's approximation: its relative
// error, at most 2^-20, is squared by each step, so that the last rounding is
// all that is left (half an ulp).  The pivot steps wait for it; a division has
// a latency of 74 cycles (B200).  The approximation takes subnormal arguments
// and results for zero: such x, to which no equilibrated system leads, are
// scaled by a power of two, by the thread that publishes the pivot row (behind
// a test of the exponent) or for all (the condensation's sweep).
#pragma once

#include <cuda_runtime.h>

namespace ddhdg
{
  // normal x with a normal reciprocal
  __device__ __forceinline__ double
  reciprocal_normal(double x)
  {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(r, fma(-x, r, 1.), r);
    r = fma(r, fma(-x, r, 1.), r);
    return r;
  }

  // the high word of |x| belongs to an x outside that range: zero, subnormal,
  // at least 2^1022 or not finite
  __device__ __forceinline__ bool
  reciprocal_special(unsigned hi)
  {
    return (hi >> 20) - 1u >= 2044u;
  }

  // such x: as 1 / x, but 0 for zero
  __device__ __forceinline__ double
  reciprocal_of_special(double x)
  {
    const double s = fabs(x) < 1. ? 0x1p64 : 0x1p-64;
    const double r = reciprocal_normal(x * s) * s;
    return x == 0. || isinf(x) ? 0. : r;
  }

  // any x, r = reciprocal_normal(x) computed before
  __device__ __forceinline__ double
  reciprocal(double x, double r)
  {
    if (reciprocal_special((unsigned)__double2hiint(x) & 0x7fffffffu))
      r = reciprocal_of_special(x);
    return r;
  }

  // Without a branch: the reciprocal of x = ReciprocalScale y with
  // |y| < 2^960, subnormal or not; 0 for x = 0, NaN where x is not finite
  constexpr double ReciprocalScale = 0x1p60;
  __device__ __forceinline__ double
  reciprocal_scaled(double x)
  {
    const double r = reciprocal_normal(x);
    return x != 0. ? r : 0.;
  }
  __device__ __forceinline__ float
  reciprocal_scaled(float x) // not scaled
  {
    return x != 0.f ? 1.f / x : 0.f;
  }
} // namespace ddhdg
