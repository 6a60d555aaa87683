// FP64 reciprocals by Newton's iteration and quotients by iterative refinement, in place of rounded
// divisions that are a few hundred cycles on a dependent chain (the pivots of the l x l factorisations)
// or a third of the arithmetic of an entry (genotype posteriors). The only rounding that
// matters is the last step's: results are the correctly rounded ones but for a few in 10^8,
// which are the value beside it.
#pragma once

namespace pg {

// 1 / x for a normal x whose reciprocal is normal: the hardware's approximation (about 20 bits) and
// two Newton steps y += y (1 - x y).
__device__ __forceinline__ double fast_reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// 1 / x for any x: zeros, NaN and values at the ends of the normal range take the division.
__device__ __forceinline__ double reciprocal(double x) {
  return x > 1e-300 && x < 1e300 ? fast_reciprocal(x) : 1.0 / x;
}

// n / x from y = 1 / x (x finite): n y and one step of refinement with its exact residual, where n y alone
// is a rounding further off. A product that is not finite is the result (x = 0, infinite and
// NaN n).
__device__ __forceinline__ double quotient(double n, double x, double y) {
  const double q = n * y;
  return fabs(q) <= 1.7976931348623157e308 ? fma(fma(-x, q, n), y, q) : q;
}

}  // namespace pg
