// FP64 reciprocal powers of a squared distance for the pair sums.
//
// Both start from the hardware's approximate reciprocal square root y of x
// (one MUFU instruction) and apply the binomial series of (1 - e)^(-1/2) and
// (1 - e)^(-3/2) in the residual e = 1 - x y^2, cut after e^2 (the third-order
// member of Householder's family of iterations).  rsqrt(x) = y (1 - e)^(-1/2)
// and x^(-3/2) = y^3 (1 - e)^(-3/2) hold exactly, so the error is the first
// dropped term, (5/16) e^3 and (35/16) e^3, plus the roundings of the last
// operations.  They take no branches and 5 and 7 FP64 operations; x must be a
// positive normal number whose y^2 and y^3 are finite, anything else gives a
// NaN, an infinity or 0, which callers that accept such inputs look for.
#pragma once

#include <cuda_runtime.h>

namespace bh {

__device__ __forceinline__ double rsqrt_approx64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// x^(-1/2)
__device__ __forceinline__ double inv_sqrt64(double x) {
  const double y = rsqrt_approx64(x);
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// m x^(-3/2)
__device__ __forceinline__ double mass_over_r3(double x, double m) {
  const double y = rsqrt_approx64(x);
  const double t = y * y;
  const double e = fma(-x, t, 1.0);
  const double w = t * (y * m);
  return fma(w * e, fma(1.875, e, 1.5), w);
}

}  // namespace bh
