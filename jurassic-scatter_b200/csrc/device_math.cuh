// Divisions by numbers that are known beforehand.
#pragma once

// num / b from the rounded reciprocal y of b, corrected by the exact
// remainder (Markstein 1990: a quotient within an ulp plus one such step is
// the rounded quotient).
__device__ __forceinline__ double div_known(double num, double b, double y) {
  const double q = num * y;
  return __fma_rn(__fma_rn(-b, q, num), y, q);
}

// jsc_lin with the width b = x1 - x0 and its reciprocal y.
__device__ __forceinline__ double lin_known(double x0, double y0, double y1, double x, double2 by) {
  return y0 + div_known(y1 - y0, by.x, by.y) * (x - x0);
}
