// The phase step's logarithm of a quotient and reciprocal square root (k_phase): branch-free FP64, so that
// the chains of a thread's two cells interleave.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace mhit {

// log(a/b) for finite b > 0 and a > 0 (a = 0: -inf, a < 0 or NaN: NaN), to two ulps, without branches,
// conversions or a separate quotient: with k the integer nearest to the difference of
// the operands' piecewise-linear log2 (exponent and mantissa fields of the high words) and
// a' = a 2^-k, a'/b lies in [0.66, 1.51] and
//   log(a/b) = k log 2 + 2 atanh(s),  s = (a' - b)/(a' + b), |s| < 0.201,
// a' - b exact (Sterbenz).  2 atanh(s) = 2 s (1 + z Q(z)), z = s^2, Q the degree-7 interpolant of
// the series 1/3 + z/5 + z^2/7 + ... at the Chebyshev nodes of [0, 0.0415] (2^-60 of the sum).
// The quotient is one Newton-Raphson step on the approximate reciprocal and one residual
// correction (Markstein); log 2 is split in two so that its products with k are exact (Cody and Waite).
template <bool POSITIVE> __device__ __forceinline__ double log_ratio(double a, double b) {
  const int ha = __double2hiint(a), hb = __double2hiint(b);
  const int k = (int)((unsigned)ha - (unsigned)hb + (1u << 19)) >> 20;
  const double as = __hiloint2double((int)((unsigned)ha - ((unsigned)k << 20)), __double2loint(a));
  const double kd = __hiloint2double(0x43380000, k ^ 0x80000000) - 6755401588539392.0;  // k as a double
  const double n = as - b, d = as + b;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = __fma_rn(__fma_rn(-d, r, 1.0), r, r);
  double s = n * r;
  s = __fma_rn(__fma_rn(-d, s, n), r, s);
  const double z = s * s;
  double q = 0.06839733963975679;
  q = __fma_rn(q, z, 0.06600187405442207);
  q = __fma_rn(q, z, 0.07694675390670448);
  q = __fma_rn(q, z, 0.09090862660038017);
  q = __fma_rn(q, z, 0.11111111603983777);
  q = __fma_rn(q, z, 0.14285714283150056);
  q = __fma_rn(q, z, 0.20000000000005075);
  q = __fma_rn(q, z, 0.3333333333333333);
  const double t = s + s;
  // log 2 in two parts, the first exact in its products with k
  const double hi = __fma_rn(kd, 0.6931471805598903, t);
  const double carry = __fma_rn(kd, 0.6931471805598903, -hi) + t;
  const double lo = __fma_rn(kd, 5.497923018708371e-14, __fma_rn(t * z, q, carry));
  const double l = hi + lo;
  if (POSITIVE) return l;
  return a > 0.0 ? l : (a == 0.0 ? -INFINITY : NAN);
}

// 1/sqrt(x) for normal x > 0 to 2^-52: the approximate reciprocal square root y and one Householder step
// of third order, y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2
__device__ __forceinline__ double rsqrt_fast(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = __fma_rn(-(x * y), y, 1.0);
  return __fma_rn(y * e, __fma_rn(0.375, e, 0.5), y);
}

}  // namespace mhit
