// FP64 natural logarithm and exponential for the matvec's kernel entries
// (near field, FP64 tensor-tile near field, on-the-fly M2L); the setup keeps
// the correctly rounded log_cr / exp_cr of exact_math.cuh.
//
// Both are table-driven (P. T. P. Tang, ACM TOMS 16(4), 1990, and 15(2),
// 1989) with tables of 32 entries only, kept as one 128-byte line per 32-bit
// word of an entry.  A warp's 32 lanes look up 32 different entries, and what
// such a gather costs is the number of lines it touches, served one after
// another by the L1 that the SM's four FP64 pipes share: the earlier tables
// (129 entries of 8 and 16 bytes, 24 lines) took ~24 L1 cycles per 32 entries
// where the ~25 FP64 operations of an entry take 13 (64 lanes per SM and
// cycle), so the FP64 near field of the log kernel was bound by its table.  A
// word line is one L1 cycle: four of them here, at the price of three more
// polynomial steps (when the tables were changed, every pair then evaluated
// twice: FP64 near field at 1,048,576 uniform points, log, 1.48 -> 1.34 ms).
#pragma once

#include "math_tables.cuh"

namespace afmm {

// ln x for positive normal x.  x = 2^k m with m in [1 - 2^-6, 2 - 2^-6), j/32
// nearest m - 1, c near 1/m of six or seven bits, so that u = m c - 1 is exact
// (make_math_tables.py: log_centre), |u| < 0.0198, c = 1 for j = 0:
//   ln x = (k ln2_hi + L_hi) + (u + (k ln2_lo + L_lo + u^2 q(u))),  L = -ln c.
// ln2_hi and L_hi are multiples of 2^-42, so the first bracket is exact for
// every exponent, and it is zero around x = 1 (j = 0, k = 0, on both sides),
// where small results keep full relative accuracy; elsewhere it is larger than
// u, and their sum's rounding error joins the small terms.  q is the truncated
// Chebyshev expansion of (ln(1+u) - u)/u^2.  17 FP64 operations.  Error below
// 0.53 ulp (tests); with c of 21 bits, a rounded u, one term less in q and u
// added to the small terms (14 operations) it was 1.2 ulp, in the form with the
// 129-entry table 0.76.  What the accuracy costs: near field at 1,048,576 points
// 0.79 -> 0.83 ms.  Zero, subnormal and non-finite inputs give an unspecified
// value without a trap, which the kernel functors select away.
__device__ __forceinline__ double log_t32(double x) {
  const int hx = __double2hiint(x);
  const int t = hx + 0x4000;  // rounds the fraction to 5 bits, carrying into the exponent
  const int j = (t >> 15) & 31;
  const double m = __hiloint2double(hx - ((t & 0xfff00000) - 0x3ff00000), __double2loint(x));
  const double kd = (double)((t >> 20) - 1023);  // (a conversion: it does not take the FP64 pipe's time)
  const unsigned int* T = &kLogT32[0][j];
  const double c = __hiloint2double((int)__ldg(T), 0);
  const double Lh = __hiloint2double((int)__ldg(T + 32), (int)__ldg(T + 64));
  const double Ll = __hiloint2double((int)__ldg(T + 96), 0);
  const double u = fma(m, c, -1.0);  // exact
  const double hi = fma(kd, kLn2Hi, Lh);  // exact
  const double lo = fma(kd, kLn2Lo, Ll);
  double q = fma(kLogQ7, u, kLogQ6);
  q = fma(q, u, kLogQ5);
  q = fma(q, u, kLogQ4);
  q = fma(q, u, kLogQ3);
  q = fma(q, u, kLogQ2);
  q = fma(q, u, kLogQ1);
  q = fma(q, u, kLogQ0);
  const double s = hi + u;
  return s + ((u - (s - hi)) + fma(q, u * u, lo));
}

// exp x.  x = (32 m + j) ln2/32 + r with N = 32 m + j the integer nearest
// x 32/ln2, j = N mod 32, |r| <= ln2/64 (r = x - N L1 - N L2, N L1 exact);
//   exp(x) = 2^m (S_hi + (S_lo + S p(r))),  S = 2^(j/32) = S_hi + S_lo,
// p(r) = exp(r) - 1 by its Taylor polynomial to r^6 (truncation below
// 2^-58); 2^m is added to the exponent bits.  13 FP64 operations.  Error at
// most 0.55 ulp for x in [-708, 709.7] (tests over that range); below -708 it
// returns 0 (the true value is under 2^-1021).
__device__ __forceinline__ double exp_t32(double x) {
  const double shifter = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
  const double t = fma(x, k32OverLn2, shifter);
  const int N = __double2loint(t);
  const double nd = t - shifter;
  double r = fma(-nd, kLn2Over32Hi, x);  // exact
  r = fma(-nd, kLn2Over32Lo, r);
  const unsigned int* T = &kExpT32[0][N & 31];
  const double Sh = __hiloint2double((int)__ldg(T), (int)__ldg(T + 32));
  const double Sl = __hiloint2double((int)__ldg(T + 64), 0);
  double q = fma(1.0 / 720.0, r, 1.0 / 120.0);
  q = fma(q, r, 1.0 / 24.0);
  q = fma(q, r, 1.0 / 6.0);
  q = fma(q, r, 0.5);
  const double p = fma(q * r, r, r);
  const double v = Sh + fma(Sh, p, fma(Sl, p, Sl));
  const double y = __hiloint2double(__double2hiint(v) + ((N >> 5) << 20), __double2loint(v));
  return x < -708.0 ? 0.0 : y;
}

// The names under which user kernels were first offered these functions.
__device__ __forceinline__ double log_tang(double x) { return log_t32(x); }
__device__ __forceinline__ double exp_tang(double x) { return exp_t32(x); }

}  // namespace afmm
