// FP64 elementary steps of the Green's-function kernels (assembly, coil fields).
// GB300 does two FP64 FMAs per clock and SM, and these kernels are bound by them:
// a kernel value needs 1/R, R and exp(-i k R) at once, which the library's sqrt,
// division and sincos give in about twice the FP64 operations of the forms here
// (arguments are moderate: no large-argument reduction, no special cases on the
// way).
#pragma once

namespace marie {

// 1/sqrt(x) and sqrt(x): FP32 estimate (bits moved by integer operations: FP64
// conversions share the FP64 pipe), one third-order Newton step (error of the
// estimate 2^-22, e^3 below 2^-60), sqrt as x times it.  Within two units in the
// last place.  Outside [1e-30, 1e30] the library functions.
__device__ __forceinline__ double inv_sqrt(double x, double& root) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  if (hi < 0x39B4484C || hi > 0x46293E59) {   // ~1e-30, ~1e30 (negative and NaN go there too)
    root = sqrt(x);
    return 1.0 / root;
  }
  const float y0 = rsqrtf(__uint_as_float((((unsigned)hi - (896u << 20)) << 3) | (lo >> 29)));
  const unsigned b = __float_as_uint(y0);
  const double y = __hiloint2double((int)((b >> 3) + (896u << 20)), (int)(b << 29));
  const double e = fma(-(x * y), y, 1.0);
  const double r = fma(y * e, fma(e, 0.375, 0.5), y);
  root = x * r;
  return r;
}

// sin and cos of |x| <= pi/4 by their Taylor polynomials (to x^15 and x^16: the
// next terms are below 5e-17), after subtracting the nearest multiple of pi/2 in
// two parts (Cody and Waite); beyond 1e4 the library function.
__device__ __forceinline__ void sin_cos(double x, double* sn, double* cs) {
  if (!(fabs(x) < 1e4)) {
    sincos(x, sn, cs);
    return;
  }
  const double magic = 6755399441055744.0;                 // 1.5 * 2^52: the sum's low word holds the integer
  const double t = fma(x, 0.63661977236758134308, magic);
  const int n = __double2loint(t);
  const double k = t - magic;
  double r = fma(-k, 1.57079632679489661923, x);
  r = fma(-k, 6.12323399573676603587e-17, r);
  const double q = r * r;
  double s = -1.0 / 1307674368000.0;
  s = fma(s, q, 1.0 / 6227020800.0);
  s = fma(s, q, -1.0 / 39916800.0);
  s = fma(s, q, 1.0 / 362880.0);
  s = fma(s, q, -1.0 / 5040.0);
  s = fma(s, q, 1.0 / 120.0);
  s = fma(s, q, -1.0 / 6.0);
  s = fma(r * q, s, r);
  double c = 1.0 / 20922789888000.0;
  c = fma(c, q, -1.0 / 87178291200.0);
  c = fma(c, q, 1.0 / 479001600.0);
  c = fma(c, q, -1.0 / 3628800.0);
  c = fma(c, q, 1.0 / 40320.0);
  c = fma(c, q, -1.0 / 720.0);
  c = fma(c, q, 1.0 / 24.0);
  c = fma(c, q, -0.5);
  c = fma(c, q, 1.0);
  const double a = (n & 1) ? c : s, b = (n & 1) ? s : c;
  *sn = __hiloint2double(__double2hiint(a) ^ ((n & 2) << 30), __double2loint(a));
  *cs = __hiloint2double(__double2hiint(b) ^ (((n + 1) & 2) << 30), __double2loint(b));
}

// sin and cos of |x| <= 0.05 (Taylor to x^7 and x^8: the next terms are below
// 6e-18).
__device__ __forceinline__ void sin_cos_small(double x, double* sn, double* cs) {
  const double q = x * x;
  *sn = fma(x * q, fma(fma(-1.0 / 5040.0, q, 1.0 / 120.0), q, -1.0 / 6.0), x);
  *cs = fma(fma(fma(fma(1.0 / 40320.0, q, -1.0 / 720.0), q, 1.0 / 24.0), q, -0.5), q, 1.0);
}

}  // namespace marie
