// Parabolic reconstruction of one zone, para_recon (reconstruct.c:142-201): the dividing form
// and the form without divisions that the sweeps run.  Plain C++ apart from the warp votes
// and the fused multiply-add, so the host can run both forms on the same inputs.
#pragma once
#include <math.h>
#include <string.h>
#include "mdg_internal.h"

#ifdef __CUDACC__
#define MDG_INLINE __forceinline__
#else
#define MDG_INLINE inline
#endif

namespace mdg {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ bool warp_all(bool b) { return __all_sync(__activemask(), b); }
__device__ __forceinline__ bool warp_any(bool b) { return __any_sync(__activemask(), b); }
__device__ __forceinline__ double fused(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ int high_word(double x) { return __double2hiint(x); }
#else
MDG_HD inline bool warp_all(bool b) { return b; }
MDG_HD inline bool warp_any(bool b) { return b; }
MDG_HD inline double fused(double a, double b, double c) { return fma(a, b, c); }
MDG_HD inline int high_word(double x)
{
  int64_t b;
  memcpy(&b, &x, 8);
  return (int)(b >> 32);
}
#endif

// para_recon for one zone (reconstruct.c:142-201): am/a0/ap are the zone averages at
// i-1, i, i+1; returns the left (al) and right (ar) face values of zone i.
//
// Control flow is arranged for the SIMT machine without changing any result: the
// extremum test (reconstruct.c:145) only skips the work when every active lane of the
// warp is at an extremum; otherwise all lanes compute and extremum lanes select a[i] at
// the end.  The two "move the zero" cases (reconstruct.c:190-200) share one code path.
// This form divides as the reference does; the sweeps run para_recon_fast and come here
// for the rare zones it declines.
template <typename T, typename G>
MDG_HD MDG_INLINE void para_recon_zone(T am_v, T a, T ap_v, const G &g, T &al, T &ar)
{
  T dqm = a - am_v;
  T dqp = ap_v - a;
  const bool flat = (dqm * dqp <= T(0));
  if (warp_all(flat)) { al = a; ar = a; return; }
  T dqc = ap_v - am_v;
  T A = (dqm * g(RC_BP) * g(RC_GM) * g(RC_G0) + g(RC_GP) * (dqp * g(RC_BM) * g(RC_G0) - dqc * g(RC_B0) * g(RC_GM))) * g(RC_DEN1);
  T B = -(dqm * g(RC_AP) * g(RC_GM) * g(RC_G0) + g(RC_GP) * (dqp * g(RC_AM) * g(RC_G0) - dqc * g(RC_A0) * g(RC_GM))) * g(RC_DEN1);
  T C = a - (g(RC_A0) * A + g(RC_B0) * B) / g(RC_G0);
  const T xl = g(RC_XL), xr = g(RC_XR);
  T l = xl * (A * xl + B) + C;
  T r = xr * (A * xr + B) + C;
  T mean = T(0.75) * am_v + T(0.25) * a;
  T mask = (a - l) * (l - mean);
  l = (mask < T(0)) ? mean : l;
  mean = T(0.75) * ap_v + T(0.25) * a;
  mask = (mean - r) * (r - a);
  r = (mask < T(0)) ? mean : r;
  A = (g(RC_B0) * (r - l) + g(RC_G0) * (a * (xl - xr) - r * xl + l * xr)) * g(RC_DEN2);
  B = (g(RC_A0) * (l - r) + g(RC_G0) * (r - a) * (xl * xl) + g(RC_G0) * (a - l) * (xr * xr)) * g(RC_DEN2);
  T xzero = -B / (T(2) * A + T(1.0e-16));
  if (isinf(xzero) || isnan(xzero)) xzero = T(-1.0e-200);
  const bool inside = !flat && (xzero > xl && xzero < xr);
  if (warp_any(inside)) {
    // move the zero to the right edge (replace al) or to the left edge (replace ar)
    const bool right = xzero > T(0.5) * (xl + xr);
    const T e = right ? r : l;
    const T xe = right ? xr : xl;
    const T xo = right ? xl : xr;
    A = g(RC_G0) * (a - e) / (right ? g(RC_DMR) : g(RC_DML));
    B = T(-2.0) * A * xe;
    C = a - (g(RC_A0) * A + g(RC_B0) * B) / g(RC_G0);
    const T val = xo * (A * xo + B) + C;
    if (inside) {
      if (right) l = val;
      else r = val;
    }
  }
  al = flat ? a : l;
  ar = flat ? a : r;
}

// a / b, correctly rounded, from y = 1/b correctly rounded: the quotient estimate a y is
// corrected twice by its remainder a - b q, which a fused multiply-add forms exactly
// (Markstein, IBM J. Res. Dev. 34, 1990: with y the rounded reciprocal and q within one
// ulp, q + (a - b q) y rounds to the quotient; the first correction puts q there).  Five
// operations without a branch.  The caller keeps a and b where no step over- or underflows
// (recon_in_range).
MDG_HD MDG_INLINE double div_by(double a, double b, double y)
{
  double q = a * y;
  q = fused(fused(-b, q, a), y, q);
  return fused(fused(-b, q, a), y, q);
}

// |x| in [2^-500, 2^500): quotients of two such numbers and their remainders are normal.
MDG_HD MDG_INLINE bool recon_in_range(double x)
{
  constexpr unsigned lo = (1023u - 500u) << 20, hi = (1023u + 500u) << 20;
  return ((unsigned)high_word(x) & 0x7fffffffu) - lo < hi - lo;
}

// para_recon of one variable: para_recon_zone's results bit for bit, with the same
// expressions, without a division and with one warp vote as its only branch.
//  * Divisions by the zone constants Gamma[i] and the two "move the zero" denominators use
//    their reciprocals from the table (div_by).
//  * The zero of the derivative, xzero = -B/D with D = 2A + 1e-16, is only compared with the
//    zone's edges and centre x: fl(-B/D) > x has the sign of e = -B - x D over that of D (one
//    fused multiply-add each, whose sign is exact) unless e is within an ulp of x of zero
//    (|e| <= |D| RC_XEPS, RC_XEPS = 2^-51 max|x|).
// Returns false where a guard fails (the caller then runs para_recon_zone): numbers outside
// recon_in_range, a zero at an edge to the last place, table constants out of range
// (RC_XEPS = inf).  The sweeps are bound by the latency of dependent FP64 operations and by
// instruction issue; measured on a B200 against the dividing form (and the quotients of
// push() by one reciprocal): FP64 400-problem ensemble 0.315 -> 0.266 ms per step, Sod 1024
// 32.2 -> 23.5 us, 384 x 128 x 256 blast 8.45 -> 7.10 ms.  Two or three variables at a time
// (interleaved streams) were slower: a variable that is constant along the direction is
// skipped alone but not beside another.
template <typename G>
MDG_HD MDG_INLINE bool para_recon_fast(double am, double a, double ap, const G &g, double &al, double &ar)
{
  const double dqm = a - am, dqp = ap - a;
  const bool flat = dqm * dqp <= 0.0;
  if (warp_all(flat)) { al = a; ar = a; return true; }
  const double dqc = ap - am;
  const double A0 = g(RC_A0), B0 = g(RC_B0), G0 = g(RC_G0), RG0 = g(RC_RG0), GM = g(RC_GM), GP = g(RC_GP);
  const double xl = g(RC_XL), xr = g(RC_XR), DEN1 = g(RC_DEN1);
  double A = (dqm * g(RC_BP) * GM * G0 + GP * (dqp * g(RC_BM) * G0 - dqc * B0 * GM)) * DEN1;
  double B = -(dqm * g(RC_AP) * GM * G0 + GP * (dqp * g(RC_AM) * G0 - dqc * A0 * GM)) * DEN1;
  double num = A0 * A + B0 * B;
  bool ok = recon_in_range(num);
  double C = a - div_by(num, G0, RG0);
  double l = xl * (A * xl + B) + C;
  double r = xr * (A * xr + B) + C;
  const double q = 0.25 * a;
  double mean = 0.75 * am + q;
  l = ((a - l) * (l - mean) < 0.0) ? mean : l;
  mean = 0.75 * ap + q;
  r = ((mean - r) * (r - a) < 0.0) ? mean : r;
  const double DEN2 = g(RC_DEN2);
  A = (B0 * (r - l) + G0 * (a * (xl - xr) - r * xl + l * xr)) * DEN2;
  B = (A0 * (l - r) + G0 * (r - a) * (xl * xl) + G0 * (a - l) * (xr * xr)) * DEN2;
  const double D = 2.0 * A + 1.0e-16, thr = fabs(D) * g(RC_XEPS), xm = 0.5 * (xl + xr);
  const double el = fused(-xl, D, -B), er = fused(-xr, D, -B), em = fused(-xm, D, -B);
  const int sD = high_word(D);
  ok = ok && recon_in_range(D) && fabs(B) < 0x1p500 && fabs(el) > thr && fabs(er) > thr && fabs(em) > thr;
  const bool inside = !flat && (high_word(el) ^ sD) >= 0 && (high_word(er) ^ sD) < 0;
  if (warp_any(inside)) {
    const bool right = (high_word(em) ^ sD) >= 0;
    const double xe = right ? xr : xl, xo = right ? xl : xr;
    num = G0 * (a - (right ? r : l));
    A = div_by(num, right ? g(RC_DMR) : g(RC_DML), right ? g(RC_RDMR) : g(RC_RDML));
    B = -2.0 * A * xe;
    const double num2 = A0 * A + B0 * B;
    ok = ok && (!inside || (recon_in_range(num) && recon_in_range(num2)));
    C = a - div_by(num2, G0, RG0);
    const double val = xo * (A * xo + B) + C;
    l = (inside && right) ? val : l;
    r = (inside && !right) ? val : r;
  }
  al = flat ? a : l;
  ar = flat ? a : r;
  return ok || flat;
}

}  // namespace mdg
