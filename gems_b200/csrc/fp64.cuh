// fp64.cuh -- branch-free FP64 functions of the pair kernels, and the SMA-TB
// pair constants they work from.
#pragma once
#include <cuda_runtime.h>
#include "common.cuh"

namespace gg {

// 1/a for normal positive a: the hardware's coarse estimate and one third-order
// step y (1 + e + e^2), e = 1 - a y (the truncated geometric series of
// 1 / (1 - e)).  The FP64 pipe runs these in a third of the instructions of
// the exact division.
__device__ __forceinline__ double rcp_pos(double a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-a, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// r = sqrt(a) and 1/r: the hardware's coarse estimate of 1/sqrt(a), one step
// of Halley's iteration, and a Newton step for r.  Branch-free, so the pairs
// of a group interleave; zero and tiny a (coincident atoms) give r ~ 0 and
// 1/r = infinity.
__device__ __forceinline__ double sqrt_pos(double a, double& rinv) {
  const bool tiny = (unsigned)__double2hiint(a) < 0x00200000u;  // a NaN of either sign is not
  a = tiny ? 1e-300 : a;
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-a * y, y, 1.0);
  y = fma(y * e, fma(0.375, e, 0.5), y);
  const double r = a * y;
  rinv = tiny ? __hiloint2double(0x7ff00000, 0) : y;
  return fma(fma(-r, r, a), 0.5 * y, r);
}

// exp(x) for |x| < EXP_MID: x = n ln 2 + f with |f| <= ln(2)/2, the Taylor
// polynomial of exp(f) to degree 13 (remainder below 5e-18), and n added to
// the exponent.  No branches (the library's exp has one for its special
// cases), so the exponentials of a group of pairs interleave: the FP64 pair
// kernels are bound by the latency of these chains, not by the FP64 rate.
constexpr double EXP_MID = 600.0;
__device__ __forceinline__ double exp_mid(double x) {
  const double big = 6755399441055744.0;  // 1.5 2^52: the sum's low word is round(x / ln 2)
  const double t = fma(x, 1.4426950408889634074, big);
  const double n = t - big;
  double f = fma(n, -0.69314718055994530942, x);
  f = fma(n, -2.3190468138462995584e-17, f);
  double p = 1.0 / 6227020800.0;
  p = fma(p, f, 1.0 / 479001600.0);
  p = fma(p, f, 1.0 / 39916800.0);
  p = fma(p, f, 1.0 / 3628800.0);
  p = fma(p, f, 1.0 / 362880.0);
  p = fma(p, f, 1.0 / 40320.0);
  p = fma(p, f, 1.0 / 5040.0);
  p = fma(p, f, 1.0 / 720.0);
  p = fma(p, f, 1.0 / 120.0);
  p = fma(p, f, 1.0 / 24.0);
  p = fma(p, f, 1.0 / 6.0);
  p = fma(p, f, 0.5);
  p = fma(p, f, 1.0);
  p = fma(p, f, 1.0);
  return __hiloint2double(__double2hiint(p) + (__double2loint(t) << 20), __double2loint(p));
}

// ------------------------------------------------------------------ SMA-TB
// Per species-pair constants of the FP64 kernels.
struct SmFP64 {
  double A, eps2, rci, rce, b1, b2, b3, r1, r2, r3;
  double p, kp, q2, kq;  // exp(-p (r/r0 - 1)) = exp(kp r + p), exp(-2q (r/r0 - 1)) = exp(kq r + q2)
  // the force pass's constants with the unit ev_ui folded in: 2 A p/r0,
  // xi^2/2 2q/r0; the tail derivatives' coefficients 5 b1, 4 b2, 3 b3 and
  // 2 (5 r1, 4 r2, 3 r3)
  double c1e, c2e, dp5, dp4, dp3, dr5, dr4, dr3;
  int wide, pad;  // the exponents leave exp_mid's range for some r <= rce
};
__host__ __device__ __forceinline__ SmFP64 sm_load(const PairP& P) {
  SmFP64 c;
  const double A = P.v[0], p = P.v[2], q = P.v[3], r0 = P.v[4], e = EV_UI;
  c.A = A;
  c.eps2 = P.v[1] * P.v[1];
  c.rci = P.v[5];
  c.rce = P.v[6];
  c.b1 = P.v[7]; c.b2 = P.v[8]; c.b3 = P.v[9];
  c.r1 = P.v[10]; c.r2 = P.v[11]; c.r3 = P.v[12];
  c.p = p;
  c.kp = -p / r0;
  c.q2 = 2.0 * q;
  c.kq = -2.0 * q / r0;
  c.c1e = 2.0 * A * p / r0 * e;
  c.c2e = c.eps2 * q / r0 * e;
  c.dp5 = 5.0 * c.b1 * e; c.dp4 = 4.0 * c.b2 * e; c.dp3 = 3.0 * c.b3 * e;
  c.dr5 = 10.0 * c.r1 * e; c.dr4 = 8.0 * c.r2 * e; c.dr3 = 6.0 * c.r3 * e;
  const double ext = fmax(fmax(fabs(p), fabs(c.q2)), fmax(fabs(fma(c.kp, c.rce, p)), fabs(fma(c.kq, c.rce, c.q2))));
  c.wide = !(ext < EXP_MID);
  c.pad = 0;
  return c;
}

// the exponentials of a pair: exp_mid inside its range, else the library's
__device__ __forceinline__ double sm_exp(const SmFP64& c, double x) { return c.wide ? exp(x) : exp_mid(x); }

}  // namespace gg
