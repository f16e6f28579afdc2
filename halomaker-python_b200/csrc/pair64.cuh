// FP64 pair arithmetic of the direct sums over a halo's members.
#pragma once
#include <cuda_runtime.h>

namespace ahop {

__device__ __forceinline__ double sep2(double dx, double dy, double dz) { return fma(dz, dz, fma(dy, dy, dx * dx)); }

// 1 / sqrt(s) for a positive normal s in five FP64 operations: the hardware's
// approximation y (rsqrt.approx.ftz.f64), then with e = 1 - s y^2 the first
// three terms of the binomial series (1 - e)^(-1/2) = 1 + e/2 + 3 e^2/8 + ...
// The next term, 5 e^3/16, is below 2^-55 for |e| < 2^-18 (y within 2^-19), less
// than a quarter of a unit in the last place; with the roundings the result is
// within two units.  s = 0 and subnormal s give NaN.
__device__ __forceinline__ double rsqrt3(double s) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  const double e = fma(-(s * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

}  // namespace ahop
