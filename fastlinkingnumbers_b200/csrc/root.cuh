// Square root of the FP64 direct sum.
#pragma once

namespace fln {

// The hardware's approximate reciprocal square root (relative error below 2^-19).
__device__ __forceinline__ double rsqrt_approx(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// sqrt(x) for normal x > 0: y from rsqrt_approx and one Householder step of third
// order on h = x y, with e = 1 - h y: sqrt(x) = h (1 + e/2 + 3/8 e^2 + O(e^3)).
// The step's remainder is below 2^-55.6 of the root, the rounding of h
// half an ulp at most, that of the result another half: within an ulp of the
// rounded square root. Five FP64 operations and no branch.
__device__ __forceinline__ double root(double x) {
  const double y = rsqrt_approx(x);
  const double h = x * y;
  const double e = fma(-h, y, 1.0);
  return fma(fma(0.375, e, 0.5), e * h, h);
}

}  // namespace fln
