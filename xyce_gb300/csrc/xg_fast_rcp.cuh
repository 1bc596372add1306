// xg_fast_rcp.cuh — the FP64 reciprocal, and square root with reciprocal, of
// the FMA load build.
//
// From the hardware's approximations (PTX rcp.approx.ftz.f64 and
// rsqrt.approx.ftz.f64, about 20 bits) one third-order step (Halley's, the
// cubic members of Householder's family; A. S. Householder, "The Numerical
// Treatment of a Single Nonlinear Equation", 1970) leaves an error of the
// seed's cube, far below double precision:
//   1/b:      e = 1 - b x,      x (1 + e + e^2)
//   1/sqrt b: e = 1 - b x^2,    x (1 + e/2 + 3 e^2/8)
// three multiply-adds for the reciprocal, which is within 2 ulp of 1.0 / b
// (tests/test_gpu_load.py, xg_probe_reciprocal); GB300 issues one in 66
// cycles, so the fourth that two Newton steps take is a quarter of the time.
// The square root is corrected by its remainder to IEEE's rounding
// (Markstein's correction) and shares its reciprocal's steps: eight FP64
// instructions for both, against 9.1 of their time for sqrt and 3 more.
// Outside the exponent ranges below (zero, subnormal, huge, infinite, NaN and
// negative operands) IEEE's own operations are used, chosen by an integer test.
#pragma once

namespace xg {

// b, opaque to the compiler: a division of it in a rarely taken branch stays
// in the branch.  (Left to itself the compiler computes the division on the
// common path too and selects: 361 cycles.)
__device__ __forceinline__ double kept_apart(double b) {
  asm volatile("mov.f64 %0, %0;" : "+d"(b));
  return b;
}

__device__ __forceinline__ double fast_rcp(double b) {
  const unsigned e = (unsigned(__double2hiint(b)) >> 20) & 0x7ffu;
  if (e - 23u > 2000u) return 1.0 / kept_apart(b);  // biased exponent outside [23, 2023]
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(b));
  const double t = fma(-b, x, 1.0);
  return fma(x, fma(t, t, t), x);
}

__device__ __forceinline__ double exact_sqrt(double b, double *r) {
  const double s = sqrt(b);
  *r = 1.0 / s;
  return s;
}

// sqrt(b), and its reciprocal in *r.
__device__ __forceinline__ double fast_sqrt(double b, double *r) {
  const unsigned e = unsigned(__double2hiint(b)) >> 20;  // sign included
  if (e - 123u > 1800u) {  // not a positive number of biased exponent [123, 1923]
    const double s = sqrt(kept_apart(b));
    *r = 1.0 / s;
    return s;
  }
  double x;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(b));
  const double h = b * x;
  const double t = fma(-h, x, 1.0);
  const double q = t * fma(0.375, t, 0.5);
  const double s = fma(h, q, h), y = fma(x, q, x);
  *r = y;
  // half of y: its exponent less one
  const double yh = __hiloint2double(__double2hiint(y) - (1 << 20), __double2loint(y));
  return fma(fma(-s, s, b), yh, s);
}

}  // namespace xg
