// A quotient whose divisor serves several: the product with the divisor's inverse, corrected once by its
// remainder. Compiles for the host too.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define LP_HD __host__ __device__ __forceinline__
#else
#define LP_HD inline
#endif

// a / b from y, 1 / b to a few roundings: correctly rounded where y is the rounded inverse (Markstein's theorem),
// within half an ulp and 1e-31 where it is the product of rounded inverses. A quotient that is not finite
// comes out a NaN.
LP_HD double lp_quotient(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-q, b, a), y, q);
}
// the same, an infinite quotient left as it is
LP_HD double lp_quotient_inf(double a, double b, double y) {
  const double q = a * y;
  return isfinite(q) ? fma(fma(-q, b, a), y, q) : q;
}
