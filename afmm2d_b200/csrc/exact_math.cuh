// Correctly rounded (to within one rounding of a ~2^-100-accurate value)
// double-precision log and exp for the setup kernels.
//
// The setup (ACA pivoting, L2P, M2L blocks) must see the same kernel entries
// as the reference's host code, whose libm log/exp return the correctly
// rounded result in all but vanishingly rare cases.  These functions evaluate
// in double-double arithmetic and round once:
//  * error-free transformations: TwoSum (Knuth), TwoProduct via FMA, and
//    double-double add / multiply / divide after Dekker (1971);
//  * log(x) = e*ln2 + 2*atanh(s), s = (m-1)/(m+1), x = m*2^e with
//    m in [1/sqrt2, sqrt2): |s| <= 0.1716, 22 odd terms of the atanh series
//    reach 2^-106;
//  * exp(x) = 2^k * exp(r), x = k*ln2 + r, |r| <= ln2/2 (r formed in
//    double-double), exp(r) by its Taylor series to 2^-106 (27 terms).
// ln 2 is carried as the double-double 0x1.62e42fefa39efp-1 + 0x1.abc9e3b39803fp-56.
//
// The double-double series (log_cr_series, exp_cr_series) cost ~1,000 FP64
// operations a call and bounded the setup: log_cr and exp_cr first evaluate a
// table-driven form to about 2^-67 (the tables of fast_math.cuh, ~45
// operations) and keep its rounding when every value within the error bound
// rounds to the same double (A. Ziv's rounding test, ACM TOMS 17(3), 1991);
// the remaining arguments (about one in 2^12) take the series, so the results
// are the series' own.  Measured on 262,144 uniform points (log, TOL 10):
// ACA 62 -> 39 ms, M2L blocks 13.2 -> 4.1 ms.
#pragma once

#include "math_tables.cuh"

namespace afmm {

struct dd {
  double hi, lo;
};

__device__ __forceinline__ dd dd_two_sum(double a, double b) {
  double s = __dadd_rn(a, b);
  double bb = __dsub_rn(s, a);
  double e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
  return dd{s, e};
}

__device__ __forceinline__ dd dd_fast_two_sum(double a, double b) {  // |a| >= |b|
  double s = __dadd_rn(a, b);
  return dd{s, __dsub_rn(b, __dsub_rn(s, a))};
}

__device__ __forceinline__ dd dd_add(dd a, dd b) {
  dd s = dd_two_sum(a.hi, b.hi);
  dd t = dd_two_sum(a.lo, b.lo);
  s.lo = __dadd_rn(s.lo, t.hi);
  s = dd_fast_two_sum(s.hi, s.lo);
  s.lo = __dadd_rn(s.lo, t.lo);
  return dd_fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ dd dd_mul(dd a, dd b) {
  double p = __dmul_rn(a.hi, b.hi);
  double e = __fma_rn(a.hi, b.hi, -p);
  e = __fma_rn(a.hi, b.lo, e);
  e = __fma_rn(a.lo, b.hi, e);
  return dd_fast_two_sum(p, e);
}

__device__ __forceinline__ dd dd_mul_d(dd a, double b) {
  double p = __dmul_rn(a.hi, b);
  double e = __fma_rn(a.hi, b, -p);
  e = __fma_rn(a.lo, b, e);
  return dd_fast_two_sum(p, e);
}

__device__ __forceinline__ dd dd_div(dd a, dd b) {
  double q1 = __ddiv_rn(a.hi, b.hi);
  dd r = dd_add(a, dd_mul_d(b, -q1));
  double q2 = __ddiv_rn(r.hi, b.hi);
  r = dd_add(r, dd_mul_d(b, -q2));
  double q3 = __ddiv_rn(r.hi, b.hi);
  dd q = dd_fast_two_sum(q1, q2);
  return dd_add(q, dd{q3, 0.0});
}

__device__ __forceinline__ dd dd_ln2() { return dd{0x1.62e42fefa39efp-1, 0x1.abc9e3b39803fp-56}; }

// 1/n for a small integer n as a double-double: h = rn(1/n), l = (1 - h*n)*h
// (the residual 1 - h*n is exact with FMA; l carries it to ~2^-106).
__device__ __forceinline__ dd dd_inv_int(double n) {
  double h = __drcp_rn(n);
  return dd{h, __dmul_rn(__fma_rn(-h, n, 1.0), h)};
}

// log(x) for finite x > 0.
static __device__ __noinline__ double log_cr_series(double x) {
  int e;
  double m = frexp(x, &e);  // x = m * 2^e, m in [0.5, 1)
  if (m < 0.70710678118654752440) {
    m = __dmul_rn(m, 2.0);
    e -= 1;
  }
  if (m == 1.0 && e == 0) return 0.0;
  dd num = dd_two_sum(m, -1.0);
  dd den = dd_two_sum(m, 1.0);
  dd s = dd_div(num, den);
  dd s2 = dd_mul(s, s);
  // atanh(s)/s = sum_{k>=0} s^(2k)/(2k+1), Horner from the tail
  dd acc = dd_inv_int(43.0);
  for (int k = 20; k >= 0; --k) acc = dd_add(dd_inv_int((double)(2 * k + 1)), dd_mul(acc, s2));
  dd lm = dd_mul(dd_mul_d(s, 2.0), acc);
  dd r = dd_add(dd_mul_d(dd_ln2(), (double)e), lm);
  return __dadd_rn(r.hi, r.lo);
}

// exp(x) for finite x (results that under/overflow follow 2^k scaling).
static __device__ __noinline__ double exp_cr_series(double x) {
  if (x == 0.0) return 1.0;
  if (x < -745.2) return 0.0;
  if (x > 709.8) return __longlong_as_double(0x7ff0000000000000LL);
  double kf = rint(x * 1.4426950408889634074);
  int k = (int)kf;
  // r = x - k*ln2 in double-double
  dd r = dd_add(dd{x, 0.0}, dd_mul_d(dd_ln2(), -kf));
  // exp(r) = sum r^n / n!, Horner from n = 27
  dd acc{1.0, 0.0};
  for (int n = 27; n >= 1; --n) acc = dd_add(dd{1.0, 0.0}, dd_mul(dd_mul(acc, r), dd_inv_int((double)n)));
  // scale by 2^k in two steps to stay normal where possible
  int k1 = k / 2, k2 = k - k1;
  double hi = __dadd_rn(acc.hi, acc.lo);
  return ldexp(ldexp(hi, k1), k2);
}

// Rounding test: true when every value within eps |hi| of hi + lo (hi = the
// rounded sum) rounds to the same double, which is then `r`.
__device__ __forceinline__ bool cr_certain(dd v, double eps, double& r) {
  const double e = fabs(v.hi) * eps;
  r = __dadd_rn(v.hi, __dadd_rn(v.lo, e));
  return r == __dadd_rn(v.hi, __dsub_rn(v.lo, e));
}

// log(x) for finite x > 0, the rounding of a value exact to 2^-100.
// x = 2^k m, F = 1 + j/128 nearest m, u = (m - F)/F = u0 + u1 (to 2^-104),
// |u| <= 2^-8:
//   ln x = (k ln2_hi + lnF_hi) + u0 - u0^2/2 + tail,
//   tail = k ln2_lo + lnF_lo + u1 (1 - u0 + u0^2) + u0^3 (1/3 - u0/4 + ... + u0^6/9),
// the three leading terms added without error (k ln2_hi + lnF_hi is exact).
// Errors relative to |u| <= |ln x| (1 + 2^-8): the cubic term's rounding
// 1.5 2^-69, the tail's additions 1.4 2^-69, truncation 2^-75: below 2^-67.
__device__ __forceinline__ double log_cr(double x) {
  const int hx = __double2hiint(x), lx = __double2loint(x);
  if ((unsigned)(hx - 0x00100000) >= 0x7fe00000u) return log_cr_series(x);  // not a positive normal number
  const int frac_hi = hx & 0x000fffff;
  const int j = (frac_hi + 0x1000) >> 13;
  const double m = __hiloint2double(frac_hi | 0x3ff00000, lx);
  const double F = __hiloint2double(0x3ff00000 + (j << 13), 0);
  const double kd = (double)((hx >> 20) - 1023);
  const double f = __dsub_rn(m, F);  // exact
  const double inv = __ldg(&kLogInvF[j]);
  const double2 lnF = __ldg(&kLogLnF[j]);
  const double hi = __fma_rn(kd, kLn2Hi, lnF.x);  // exact
  const double u0 = __dmul_rn(f, inv);
  const double u1 = __dmul_rn(__fma_rn(-u0, F, f), inv);
  const double hu = __dmul_rn(0.5, u0);
  const double h0 = __dmul_rn(u0, hu);
  const double h1 = __fma_rn(u0, hu, -h0);
  double q = __fma_rn(1.0 / 9.0, u0, -1.0 / 8.0);
  q = __fma_rn(q, u0, 1.0 / 7.0);
  q = __fma_rn(q, u0, -1.0 / 6.0);
  q = __fma_rn(q, u0, 1.0 / 5.0);
  q = __fma_rn(q, u0, -0.25);
  q = __fma_rn(q, u0, 1.0 / 3.0);
  const double p3 = __dmul_rn(q, __dmul_rn(u0, __dmul_rn(u0, u0)));
  const double w1 = __fma_rn(__fma_rn(u0, u0, -u0), u1, u1);
  const dd a = dd_two_sum(hi, u0);
  const dd b = dd_two_sum(a.hi, -h0);
  const double tail = __dadd_rn(__dadd_rn(a.lo, b.lo),
                                __dadd_rn(__dsub_rn(__dadd_rn(__fma_rn(kd, kLn2Lo, lnF.y), w1), h1), p3));
  double r;
  if (cr_certain(dd_fast_two_sum(b.hi, tail), 0x1p-66, r)) return r;
  return log_cr_series(x);
}

// exp(x), the rounding of a value exact to 2^-100.  x = (32 m + j) ln2/32 + r,
// r = r0 + r1 (to 2^-82), |r| <= ln2/64, S = 2^(j/32) = S_hi + S_lo:
//   exp(x) = 2^m S (1 + P),  P = r0 + r0^2/2 + tail,
//   tail = r1 (1 + r0) + r0^3 (1/6 + ... + r0^5/40320).
// Errors relative to the result: the cubic term's rounding 2^-73, the
// additions of the tails 3 2^-73.6 + 2^-72.2, truncation 2^-77: below 2^-70.
__device__ __forceinline__ double exp_cr(double x) {
  if (!(fabs(x) <= 700.0)) return exp_cr_series(x);  // the result may be subnormal or overflow
  const double shifter = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
  const double t = __fma_rn(x, k32OverLn2, shifter);
  const int N = __double2loint(t);
  const double nd = __dsub_rn(t, shifter);
  const double rh = __fma_rn(-nd, kLn2Over32Hi, x);  // exact
  const double p = __dmul_rn(nd, kLn2Over32Lo);
  const dd rr = dd_two_sum(rh, -p);
  const double r0 = rr.hi;
  const double r1 = __dsub_rn(rr.lo, __fma_rn(nd, kLn2Over32Lo, -p));
  const double hr = __dmul_rn(0.5, r0);
  const double h0 = __dmul_rn(r0, hr);
  const double h1 = __fma_rn(r0, hr, -h0);
  double q = __fma_rn(1.0 / 40320.0, r0, 1.0 / 5040.0);
  q = __fma_rn(q, r0, 1.0 / 720.0);
  q = __fma_rn(q, r0, 1.0 / 120.0);
  q = __fma_rn(q, r0, 1.0 / 24.0);
  q = __fma_rn(q, r0, 1.0 / 6.0);
  const double p3 = __dmul_rn(q, __dmul_rn(r0, __dmul_rn(r0, r0)));
  const dd P = dd_fast_two_sum(r0, h0);
  const double tail = __dadd_rn(__dadd_rn(__dadd_rn(P.lo, h1), __fma_rn(r0, r1, r1)), p3);
  const double2 S = __ldg(&kExp2J32[N & 31]);
  const double a0 = __dmul_rn(S.x, P.hi);
  const double a1 = __fma_rn(S.x, P.hi, -a0);
  const dd s = dd_fast_two_sum(S.x, a0);
  const double t2 = __dadd_rn(s.lo, __dadd_rn(a1, __fma_rn(S.x, tail, __fma_rn(S.y, P.hi, S.y))));
  double r;
  if (!cr_certain(dd_fast_two_sum(s.hi, t2), 0x1p-68, r)) return exp_cr_series(x);
  return r * __hiloint2double(((N >> 5) + 1023) << 20, 0);  // 2^m: exact
}

}  // namespace afmm
