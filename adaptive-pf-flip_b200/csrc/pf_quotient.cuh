// pf_quotient.cuh -- r / d from a stored reciprocal, with the division's bits.
//
// inv = RN(1 / d) is formed once per solve; the quotient is the product and two
// residual corrections (Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990: with a correctly rounded
// reciprocal the correction of a faithful quotient is correctly rounded; the first
// correction makes the product faithful).  Every step is exact enough only while
// nothing nears the ends of the exponent range, so a cell whose d is outside
// 2^+-400 has inv = 0, and that or an r outside 2^+-500 takes the division.  Five
// dependent operations without a branch, where the division's take the throughput
// of about 13.  Compiles for the host too, where its bits are tested.
#pragma once

#include <cmath>

namespace pf {

#ifdef __CUDACC__
#define PF_QUOTIENT_FN __device__ __forceinline__
PF_QUOTIENT_FN double q_div(double a, double b) { return __ddiv_rn(a, b); }
PF_QUOTIENT_FN double q_mul(double a, double b) { return __dmul_rn(a, b); }
PF_QUOTIENT_FN double q_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
#define PF_QUOTIENT_FN inline
PF_QUOTIENT_FN double q_div(double a, double b) { return a / b; }
PF_QUOTIENT_FN double q_mul(double a, double b) { return a * b; }
PF_QUOTIENT_FN double q_fma(double a, double b, double c) { return std::fma(a, b, c); }
#endif

PF_QUOTIENT_FN double inv_of(double d) { return d > 0x1p-400 && d < 0x1p400 ? q_div(1.0, d) : 0.0; }
PF_QUOTIENT_FN double quotient(double r, double d, double inv) {
  const double ar = std::fabs(r);
  if (!(inv != 0.0 && ((ar > 0x1p-500 && ar < 0x1p500) || ar == 0.0))) return d > 0.0 ? q_div(r, d) : 0.0;
  double q = q_mul(r, inv);
  // the residuals as q d - r: with r - q d, r = -0 would end at +0
  q = q_fma(-q_fma(q, d, -r), inv, q);
  return q_fma(-q_fma(q, d, -r), inv, q);
}
#undef PF_QUOTIENT_FN

}  // namespace pf
