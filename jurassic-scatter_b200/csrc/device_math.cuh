// Divisions by numbers that are known beforehand.
#pragma once

// num / b from the rounded reciprocal y of b, corrected by the remainder
// (Markstein 1990: one such step makes a quotient within an ulp the rounded
// one).  The first product may be off by more than an ulp, by less than two at
// the top of a binade, which the theorem does not cover; 2e9 quotients, many of
// them there or at a power of two, were those of the division.  Callers keep
// num and num / b finite and above 1e-290 or 0 (an infinite num gives NaN, a
// negative zero a positive one): steps and direction components of a march, in
// km, refractivities, emissivities in [0, 1], Riccati-Bessel functions below
// the order where they leave the range of a double.
__device__ __forceinline__ double div_known(double num, double b, double y) {
  const double q = num * y;
  return __fma_rn(__fma_rn(-b, q, num), y, q);
}

// jsc_lin with the width b = x1 - x0 and its reciprocal y.
__device__ __forceinline__ double lin_known(double x0, double y0, double y1, double x, double2 by) {
  return y0 + div_known(y1 - y0, by.x, by.y) * (x - x0);
}
