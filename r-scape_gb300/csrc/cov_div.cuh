// cov_div.cuh -- FP64 quotients in fewer instructions than the general
// division takes (this chip issues an FP64 instruction of a warp every ~64
// cycles): an approximate or shared reciprocal and corrections of the quotient
// with exact FMA residuals (Markstein, IBM J. Res. Dev. 34, 1990).
#pragma once
#include <cstdint>

namespace covgpu {

// x / b, |b| and |x| within div_range: the hardware's approximate reciprocal
// (20 bits), one third-order Newton step and one residual correction of the
// quotient: six FP64 instructions.  The corrected quotient is the IEEE one
// unless the reciprocal is the second nearest number to 1 / b (one in ~100) and
// x / b lies within 2^-105 of the middle of two numbers: then it may be the
// other neighbour (none of 40,000 such pairs was).  Just below a power of two
// both are common (1 / b is near a middle itself), so such divisors, one in a
// million, take the general division.
__device__ __forceinline__ double div_fast(double x, double b) {
  if ((__double2hiint(b) & 0xfffff) == 0xfffff) return x / b;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
  double e = __fma_rn(-b, r, 1.0);
  e = __fma_rn(e, e, e);
  r = __fma_rn(r, e, r);
  const double q = __dmul_rn(x, r);
  return __fma_rn(__fma_rn(-q, b, x), r, q);
}
__device__ __forceinline__ bool div_range(double x) {   // ~1e-30 .. 1e30, either sign
  return (unsigned)((__double2hiint(x) & 0x7fffffff) - 0x39b4484c) < (unsigned)(0x46293e59 - 0x39b4484c);
}

// x / b correctly rounded from y = 1 / b correctly rounded: a quotient within
// two ulps and two residual steps (a faithful quotient plus one such step is the
// correctly rounded one).  Five FP64 operations where the reciprocal is shared.
// Finite x and b well inside the exponent range.
__device__ __forceinline__ double div_by(double x, double b, double y) {
  double q = __dmul_rn(x, y);
  q = __fma_rn(__fma_rn(-q, b, x), y, q);
  return __fma_rn(__fma_rn(-q, b, x), y, q);
}

}  // namespace covgpu
