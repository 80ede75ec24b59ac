// 3-D spherical sweep on the dendritic grid (plain FP64, the reference's operation order).
//
// prim_to_fluxes3 (step.c:1088-1430) visits every zone once and does, in that order, its
// lower direction-0 face, its lower direction-1 face(s) and its lower direction-2 face;
// push (step.c:327-478) then differences the stored face fluxes with the dendritic
// fan-in.  Here each of the three face families is one kernel (one thread per face, the
// faces of a row (i, j) in 128-face tiles), the fluxes go to HBM, and a fourth kernel
// applies push() per zone.  What the serial order of the reference decides is kept:
//
//  * pencils.  A direction-0 face of zone (i, j, k) reads radial zones i-2 .. i+1 at the
//    face's own (theta, phi) resolution: a finer row is restricted (volume-weighted mean,
//    restrict0 step.c:1012-1051; its Gamma slot takes the zone's phi velocity, as
//    restrict0 reads p[..][GAMMA] = p[..][U3]), a coarser or equal row is prolonged by
//    limited slopes in phi and then theta (prolongate0/kslopes0, step.c:905-955, 782-840).
//    Direction-1 faces restrict/prolong across phi-refinement steps (restrict1,
//    prolongate1/kslopes1, step.c:1053-1085, 957-1010, 842-900).
//  * boundaries.  Ghost zones are not stored: a read of a ghost zone is mapped to the
//    interior zone reset_boundaries_gpu copies into it (bc.c:705-1422, i-boundaries on
//    interior (j, k), j-boundaries on interior (i, k), k-boundaries on interior (i, j));
//    ghost zones that no boundary loop writes (corners) hold zeros, as the zero-filled
//    allocation does (utils.c:164-174).
//  * shock flags.  A direction-1 or -2 face uses HLLE next to a direction-0 shock
//    (transverse_shock, fluid.c:189-210) with the flags the serial loop has set when it
//    reaches the face: ghost flags are always "shock" (never reset), the current stage
//    contributes only the zone's own direction-0 face (marks from rows i+1, i+2 come
//    later in the loop), and in the second stage every first-stage mark counts
//    (set_shock_flag(0) resets once per step).  own[c]: zone c's own face in the current
//    stage; all0[c]: any first-stage mark of zone c (faces i, i+1, i+2 map down to it).
//  * the polar-axis fix (step.c:1301-1401): on the last theta row of every radial row
//    the phi-face states are the zone values with the velocity rotated through
//    Cartesian components (host tables of the sines and cosines).
#pragma once
#include "mdg_hydro.cuh"
#include "mdg_kernels.cuh"
#include "mdg_grid3d.cuh"
#include "mdg_mixed.cuh"

namespace mdg {

struct Tile3 { int i, j, k0, cnt; };
constexpr int NT3 = 128;
// resident CTAs per SM requested from the compiler (register caps).  The face kernels wait
// on dependent gathers and on FP64 latency; ms per step on a B200 with 8 / 6 / 5 / 4 CTAs of
// 128 threads (64 / 80 / 96 / 128 registers): plain FP64 384 x 128 x 256 6.95 / 6.62 / 6.75 /
// 7.37, 128 x 64 x 128 1.37 / 1.24 / 1.47 / 1.46; mixed 384 x 128 x 256 with 8 / 7 / 6 / 5 / 4
// 5.41 / 5.27 / 5.31 / 5.44 / 5.91.
#ifndef MDG_F3MINB
#define MDG_F3MINB 6
#endif
#ifndef MDG_F3MINB_MIX
#define MDG_F3MINB_MIX 7
#endif
// Launches of at most F3MINB_SMALL CTAs per SM are all resident with 96 registers a thread as
// well, which leaves fewer spills on the chain of one thread's operations: 2-D 400 x 256 blast,
// 725 CTAs, plain FP64 202 -> 187 us per step, mixed 203 -> 164 us (384 x 128 x 256 with them: 6.69 ->
// 6.86 ms, mixed 5.25 -> 5.46).
constexpr int F3MINB_SMALL = 5;
constexpr int f3_minb(bool mix, bool small) { return small ? F3MINB_SMALL : mix ? MDG_F3MINB_MIX : MDG_F3MINB; }
#ifndef MDG_P3MINB
#define MDG_P3MINB 8
#endif

__device__ __forceinline__ int rowi(const Grid3 &g, int i, int j) { return __ldg(g.rowbase + i + NG) + j + NG; }
__device__ __forceinline__ int nj_of(const Grid3 &g, int i) { return __ldg(g.nj + i + NG); }
__device__ __forceinline__ int djs(const Grid3 &g, int i) { return g.n2 / nj_of(g, i); }
__device__ __forceinline__ int nk_of(const Grid3 &g, int i, int j) { return __ldg(g.nk + rowi(g, i, j)); }
__device__ __forceinline__ int dks(const Grid3 &g, int i, int j) { return g.n3 / nk_of(g, i, j); }
__device__ __forceinline__ double geo3(const Grid3 &g, int f, int ij) { return __ldg(g.geo + (int64_t)f * g.nij + ij); }
__device__ __forceinline__ double minmod(double a, double b)
{
  // MINMOD, decs.h:629-630
  return 0.5 * ((a < 0.0 ? -1.0 : 1.0) + (b < 0.0 ? -1.0 : 1.0)) * (fabs(a) < fabs(b) ? fabs(a) : fabs(b));
}

// Interior zone that reset_boundaries_gpu copies into zone (i, j, k), with the velocity
// components it negates (bit v set: component v flips sign); -1: a zone no boundary
// loop writes (zero).
static __device__ int64_t locate3(const Grid3 &g, int i, int j, int k, int &flip)
{
  flip = 0;
  const int n1 = g.n1;
  const bool ig = (i < 0 || i >= n1);
  const int nji = nj_of(g, i);
  const bool jg = (j < 0 || j >= nji);
  const int nkr = nk_of(g, i, j);
  const bool kg = (k < 0 || k >= nkr);
  int ip = i, jp = j, kp = k;
  if (!ig && !jg && !kg) return __ldg(g.cell + rowi(g, i, j)) + k;
  if (ig && !jg && !kg) {
    if (i < 0) {
      ip = -1 - i;
      if (g.bc_lo0 == BC_SPHERICAL_ORIGIN) {
        const int njp = g.n2 / djs(g, ip);
        jp = njp - 1 - j;
        const int nkp = g.n3 / dks(g, ip, jp);
        kp = (k + nkp / 2) % nkp;
        flip = (1 << U1) | (1 << U3);
      } else {   // REFLECT
        jp = j * djs(g, i) / djs(g, ip);
        kp = k * dks(g, i, j) / dks(g, ip, jp);
        flip = 1 << U1;
      }
    } else {
      if (g.bc_hi0 == BC_REFLECT) {
        ip = 2 * n1 - i - 1;
        flip = 1 << U1;
      } else {   // OUTFLOW
        ip = n1 - 1;
      }
    }
  } else if (!ig && jg && !kg) {
    const int bc = (j < 0) ? g.bc_lo1 : g.bc_hi1;
    if (bc == BC_OUTFLOW) {
      jp = (j < 0) ? 0 : nji - 1;
    } else {
      jp = (j < 0) ? -1 - j : 2 * nji - 1 - j;
      if (bc == BC_SPHERICAL_ORIGIN) {
        const int nkp = g.n3 / dks(g, i, jp);
        kp = (k + nkp / 2) % nkp;
        flip = (1 << U2) | (1 << U3);
      } else {   // REFLECT
        kp = k * dks(g, i, j) / dks(g, i, jp);
        flip = 1 << U2;
      }
    }
  } else if (!ig && !jg && kg) {
    const int bc = (k < 0) ? g.bc_lo2 : g.bc_hi2;
    if (bc == BC_PERIODIC) {
      kp = (k < 0) ? k + nkr : k - nkr;
    } else {
      kp = (k < 0) ? 0 : nkr - 1;
      if (bc == BC_REFLECT) flip = 1 << U3;
    }
  } else {
    return -1;
  }
  // a source outside the interior (boundary kinds that assume no refinement next to the
  // boundary, used on a grid that has some there) reads as an unwritten zone
  if (ip < 0 || ip >= n1 || jp < 0 || jp >= nj_of(g, ip) || kp < 0 || kp >= nk_of(g, ip, jp)) return -1;
  return __ldg(g.cell + rowi(g, ip, jp)) + kp;
}

// Zone (i, j, k) as the pencils see it: primitives, PRESS and GAMMA of its EOS record
// (update_eos / update_eos_ghost fill every zone, eos.c:4-34).
__device__ __forceinline__ void load7(const Grid3 &g, const ProbDev &P, const StateSoA &s, int i, int j, int k,
                                      double *w)
{
  int flip;
  const int64_t c = locate3(g, i, j, k, flip);
#pragma unroll
  for (int v = 0; v < NPRIM; v++) {
    double x = (c >= 0) ? s.v[v][c] : 0.0;
    w[v] = ((flip >> v) & 1) ? -x : x;
  }
  w[5] = eos_press(P.eos, P.gam, P.Kpoly, w[RHO], w[UU]);
  w[6] = P.gam;
}

// load7 of interior zone c; true when a value is -0 (see pencil0).
__device__ __forceinline__ bool load7_zone(const ProbDev &P, const StateSoA &s, int64_t c, double *w)
{
  bool neg0 = false;
#pragma unroll
  for (int v = 0; v < NPRIM; v++) w[v] = s.v[v][c];
  w[5] = eos_press(P.eos, P.gam, P.Kpoly, w[RHO], w[UU]);
  w[6] = P.gam;
#pragma unroll
  for (int v = 0; v < 6; v++) neg0 = neg0 || (w[v] == 0.0 && signbit(w[v]));
  return neg0;
}

// kslopes0 / kslopes1: limited phi slope of row (ii, jj) evaluated at the centroid x2p.
static __device__ void kslope_point(const Grid3 &g, const ProbDev &P, const StateSoA &s, int ii, int jj, int kk,
                             double x2p, double *pp)
{
  const int lev = ilog2(dks(g, ii, jj));
  const int base = g.rc2_base[lev] + NG;
  const double x20 = __ldg(g.xc2 + base + kk - 1), x21 = __ldg(g.xc2 + base + kk), x22 = __ldg(g.xc2 + base + kk + 1);
  const double idx2m = 1.0 / (x21 - x20), idx2p = 1.0 / (x22 - x21), idx2c = 1.0 / (x22 - x20);
  double a[7], b[7], c[7];
  load7(g, P, s, ii, jj, kk - 1, a);
  load7(g, P, s, ii, jj, kk, b);
  load7(g, P, s, ii, jj, kk + 1, c);
#pragma unroll
  for (int v = 0; v < 7; v++) {
    const double sm = (b[v] - a[v]) * idx2m;
    const double sp = (c[v] - b[v]) * idx2p;
    const double sc = (c[v] - a[v]) * idx2c;
    const double sg = minmod(2.0 * minmod(sm, sp), sc);
    pp[v] = b[v] + sg * (x2p - x21);
  }
}

// Pencil entry of radial row ii for the direction-0 face of zone (i, j, k).
static __device__ void pencil0(const Grid3 &g, const ProbDev &P, const StateSoA &s, int i, int j, int k, int ii, double *pp)
{
  const int dji = djs(g, i), djii = djs(g, ii);
  if (djii < dji) {
    // restrict0 (step.c:1012-1051)
    const int njp = dji / djii, jp = j * njp;
    const int dkij = dks(g, i, j);
    double vol_sum = 0.0;
    for (int jj = jp; jj < jp + njp; jj++) {
      const int nkp = dkij / dks(g, ii, jj);
      const double vol = geo3(g, G3_VOL, rowi(g, ii, jj));
      for (int kk = k * nkp; kk < k * nkp + nkp; kk++) vol_sum += vol;
    }
    vol_sum = 1.0 / vol_sum;
#pragma unroll
    for (int v = 0; v < 7; v++) pp[v] = 0.0;
    for (int jj = jp; jj < jp + njp; jj++) {
      const int nkp = dkij / dks(g, ii, jj);
      const double vol = geo3(g, G3_VOL, rowi(g, ii, jj));
      for (int kk = k * nkp; kk < k * nkp + nkp; kk++) {
        const double vol_frac = vol * vol_sum;
        double w[7];
        load7(g, P, s, ii, jj, kk, w);
#pragma unroll
        for (int v = 0; v < NPRIM; v++) pp[v] += w[v] * vol_frac;
        pp[5] += w[5] * vol_frac;
        pp[6] += w[U3] * vol_frac;   // p[..][GAMMA], GAMMA = 4 (decs.h:661)
      }
    }
    return;
  }
  // prolongate0 (step.c:905-955)
  if (djii == dji && dks(g, ii, j) == dks(g, i, j)) {
    // same theta and phi level: both slope corrections are multiplied by an exact +0
    // (the prolongation point is the zone's own centroid), so the result is the zone
    // value itself unless that value is -0 (then the sign of the slope decides the sign
    // of the zero sum, and the full computation below runs)
    load7(g, P, s, ii, j, k, pp);
    bool neg0 = false;
#pragma unroll
    for (int v = 0; v < 7; v++) neg0 = neg0 || (pp[v] == 0.0 && signbit(pp[v]));
    if (!neg0) return;
  }
  const int jj = j * dji / djii;
  const double x1p = __ldg(g.xc1 + g.rc1_base[ilog2(dji)] + NG + j);
  const double x2p = __ldg(g.xc2 + g.rc2_base[ilog2(dks(g, i, j))] + NG + k);
  const int dkij = dks(g, i, j);
  double p0[7], p1[7], p2[7];
  if (g.ndim == 2) {
    // the 2-D prolongate0 (step.c:579-628) has no phi slopes
    load7(g, P, s, ii, jj - 1, 0, p0);
    load7(g, P, s, ii, jj, 0, p1);
    load7(g, P, s, ii, jj + 1, 0, p2);
  } else {
    kslope_point(g, P, s, ii, jj - 1, k * dkij / dks(g, ii, jj - 1), x2p, p0);
    kslope_point(g, P, s, ii, jj, k * dkij / dks(g, ii, jj), x2p, p1);
    kslope_point(g, P, s, ii, jj + 1, k * dkij / dks(g, ii, jj + 1), x2p, p2);
  }
  const int base = g.rc1_base[ilog2(djii)] + NG;
  const double x10 = __ldg(g.xc1 + base + jj - 1), x11 = __ldg(g.xc1 + base + jj), x12 = __ldg(g.xc1 + base + jj + 1);
  const double idx1m = 1.0 / (x11 - x10), idx1p = 1.0 / (x12 - x11), idx1c = 1.0 / (x12 - x10);
#pragma unroll
  for (int v = 0; v < 7; v++) {
    const double sm = (p1[v] - p0[v]) * idx1m;
    const double sp = (p2[v] - p1[v]) * idx1p;
    const double sc = (p2[v] - p0[v]) * idx1c;
    const double sg = minmod(2.0 * minmod(sm, sp), sc);
    pp[v] = p1[v] + sg * (x1p - x11);
  }
}

// Pencil entry of theta row jj for the direction-1 sub-face kk of face row (i, j).
static __device__ void pencil1(const Grid3 &g, const ProbDev &P, const StateSoA &s, int i, int j, int kk, int jj,
                        double *pp)
{
  const int dkj = dks(g, i, j), dkjm = dks(g, i, j - 1);
  const int mn = dkj < dkjm ? dkj : dkjm;
  const int dkjj = dks(g, i, jj);
  if (dkjj < mn) {
    // restrict1 (step.c:1053-1085)
    const int nkp = mn / dkjj, kp = kk * nkp;
    const double vol = geo3(g, G3_VOL, rowi(g, i, jj));
    double vol_sum = 0.0;
    for (int k = kp; k < kp + nkp; k++) vol_sum += vol;
    vol_sum = 1.0 / vol_sum;
#pragma unroll
    for (int v = 0; v < 7; v++) pp[v] = 0.0;
    for (int k = kp; k < kp + nkp; k++) {
      const double vol_frac = vol * vol_sum;
      double w[7];
      load7(g, P, s, i, jj, k, w);
#pragma unroll
      for (int v = 0; v < 7; v++) pp[v] += w[v] * vol_frac;
    }
    return;
  }
  // prolongate1 (step.c:957-1010)
  const int k2 = kk * mn / dkjj;
  if (mn == dkjj) {
    load7(g, P, s, i, jj, k2, pp);
    return;
  }
  const double x2p = __ldg(g.xc2 + g.rc2_base[ilog2(mn)] + NG + kk);
  kslope_point(g, P, s, i, jj, k2, x2p, pp);
}

// Wave-speed estimate with per-side Gamma (riemann.c:368-429 / 210-303): the pencils of
// the dendritic grid can carry a reconstructed Gamma slot that differs between sides.
__device__ __forceinline__ void wave_speeds_g(const double *pl, const double *pr, double u_l, double u_r, bool hlle,
                                              double &sl, double &sr, double &ss, double &p_s, int &isshock)
{
  const double p_l = pl[5], p_r = pr[5], G_l = pl[6], G_r = pr[6];
  const double cs_l = sqrt(G_l * p_l / pl[RHO]);
  const double cs_r = sqrt(G_r * p_r / pr[RHO]);
  double p_max, p_min;
  if (p_l > p_r) { p_max = p_l; p_min = p_r; } else { p_max = p_r; p_min = p_l; }
  bool below2;
  pressure_ratio_tests(p_max, p_min, below2, isshock);
  p_s = 0.5 * (p_l + p_r) - 0.125 * (u_r - u_l) * (pl[RHO] + pr[RHO]) * (cs_l + cs_r);
  if (hlle) p_s = (p_s > 0.0) ? p_s : 0.0;
  else p_s = (0.0 > p_s) ? 0.0 : p_s;
  if (below2 && p_s >= p_min && p_s <= p_max) {
  } else if (p_s < p_min) {
    const double G_avg = 0.5 * (G_l + G_r);
    const double plr = pow(p_l / p_r, (G_avg - 1.0) / (2.0 * G_avg));
    const double s0 = (plr * u_l / cs_l + u_r / cs_r + 2.0 * (plr - 1.0) / (G_avg - 1.0)) / (plr / cs_l + 1.0 / cs_r);
    p_s = 0.5 * (p_l * pow(1.0 + (G_l - 1.0) / (2.0 * cs_l) * (u_l - s0), 2.0 * G_l / (G_l - 1.0))
               + p_r * pow(1.0 + (G_r - 1.0) / (2.0 * cs_r) * (s0 - u_r), 2.0 * G_r / (G_r - 1.0)));
    p_s = (p_s > 0.0) ? p_s : 0.0;
  } else {
    const double a_l = 2.0 / ((G_l + 1.0) * pl[RHO]);
    const double a_r = 2.0 / ((G_r + 1.0) * pr[RHO]);
    const double b_l = (G_l - 1.0) / (G_l + 1.0) * p_l;
    const double b_r = (G_r - 1.0) / (G_r + 1.0) * p_r;
    const double g_l = sqrt(a_l / (p_s + b_l));
    const double g_r = sqrt(a_r / (p_s + b_r));
    p_s = (g_l * p_l + g_r * p_r - (u_r - u_l)) / (g_l + g_r);
    p_s = (p_s > 0.0) ? p_s : 0.0;
  }
  const double q_l = (p_s <= p_l) ? 1.0 : sqrt(1.0 + (G_l + 1.0) / (2.0 * G_l) * (p_s / p_l - 1.0));
  const double q_r = (p_s <= p_r) ? 1.0 : sqrt(1.0 + (G_r + 1.0) / (2.0 * G_r) * (p_s / p_r - 1.0));
  sl = u_l - cs_l * q_l;
  sr = u_r + cs_r * q_r;
  ss = (p_r - p_l + pl[RHO] * u_l * (sl - u_l) - pr[RHO] * u_r * (sr - u_r))
     / (pl[RHO] * (sl - u_l) - pr[RHO] * (sr - u_r));
}

// The wave speeds of a face (riemann_flux_HLLC / HLLE, riemann.c:328-499 / 178-325, with
// per-side Gamma).
struct Waves3 { double u_l, u_r, sl, sr, ss, p_s; };

// The HLLC flux from the wave speeds.
template <int DIR>
__device__ __forceinline__ void hllc3_flux(const double *pl, const double *pr, const FaceGeom<double> &g, Waves3 w,
                                           double *flux, double &sig)
{
  const double sc = g.scale;
  if (w.ss > w.sr) w.sr = 1.001 * w.ss;
  if (w.ss < w.sl) w.sl = 1.001 * w.ss;
  sig = tmax(fabs(w.sl), fabs(w.sr)) / sc;
  if (w.sl > 0.0) { pflux<DIR, false, double>(pl, pl[5], g, flux); return; }
  if (w.sr < 0.0) { pflux<DIR, false, double>(pr, pr[5], g, flux); return; }
  double u[NPRIM], fx[NPRIM], Us[NPRIM], pk[6];
  const bool left = w.ss > 0.0;
#pragma unroll
  for (int v = 0; v < 6; v++) pk[v] = left ? pl[v] : pr[v];
  const double sk = left ? w.sl : w.sr;
  const double uk = left ? w.u_l : w.u_r;
  p_uflux<DIR, false, double>(pk, g, pk[5], u, fx);
  Us[0] = pk[RHO] * (sk - uk) / (sk - w.ss);
  Us[UU] = (u[UU] * (sk - uk) - pk[5] * uk + w.p_s * w.ss) / (sk - w.ss);
  Us[U1] = pk[U1]; Us[U2] = pk[U2]; Us[U3] = pk[U3];
  Us[U1 + DIR] = w.ss / sc;
  const double slr = sk / sc;
  const double vc0 = g.g0 * Us[U1], vc1 = g.g1 * Us[U2], vc2 = g.g2 * Us[U3];
  Us[U1] = vc0 * Us[0]; Us[U2] = vc1 * Us[0]; Us[U3] = vc2 * Us[0];
#pragma unroll
  for (int v = 0; v < NPRIM; v++) flux[v] = g.area * (fx[v] + slr * (Us[v] - u[v]));
}

// The HLLE flux from the wave speeds.
template <int DIR, bool MIX>
__device__ __forceinline__ void hlle3_flux(const double *pl, const double *pr, const FaceGeom<double> &g,
                                           const Waves3 &w, double *flux, double &sig)
{
  const double sc = g.scale;
  double ul[NPRIM], ur[NPRIM], fl[NPRIM], fr[NPRIM];
  p_uflux<DIR, false, double>(pl, g, pl[5], ul, fl);
  p_uflux<DIR, false, double>(pr, g, pr[5], ur, fr);
  const double cmax = tmax(w.sr / sc, 0.0);
  const double cmin = fabs(tmin(w.sl / sc, 0.0));
  sig = tmax(cmax, cmin);
  double num[NPRIM], q[NPRIM];
#pragma unroll
  for (int v = 0; v < NPRIM; v++) num[v] = g.area * (cmin * fr[v] + cmax * fl[v] - cmax * cmin * (ur[v] - ul[v]));
  quotients<NPRIM, MIX>(num, cmax + cmin, q);
#pragma unroll
  for (int v = 0; v < NPRIM; v++) flux[v] = q[v];
}

// FP64 solve of a face by either solver; returns isshock.  The wave speeds are the same but for
// a NaN clamp, so the lanes of a warp that take different solvers share them, and the kernels
// hold them once (instruction fetch was the second stall of face2_kernel): 128 x 64 x 128 blast,
// plain FP64, 1.37 -> 1.24 ms per step.
template <int DIR, bool MIX = false>
__device__ __forceinline__ int riemann3(bool hlle, const double *pl, const double *pr, const FaceGeom<double> &g,
                                        double *flux, double &sig)
{
  if (g.area < 1.0e-16) {
    sig = 1.0e-200;
#pragma unroll
    for (int v = 0; v < NPRIM; v++) flux[v] = 0.0;
    return 0;
  }
  Waves3 w;
  int isshock = 0;
  w.u_l = pl[U1 + DIR] * g.scale;
  w.u_r = pr[U1 + DIR] * g.scale;
  wave_speeds_g(pl, pr, w.u_l, w.u_r, hlle, w.sl, w.sr, w.ss, w.p_s, isshock);
  if (hlle) hlle3_flux<DIR, MIX>(pl, pr, g, w, flux, sig);
  else hllc3_flux<DIR>(pl, pr, g, w, flux, sig);
  return isshock;
}
template <int DIR>
__device__ __forceinline__ int hllc3(const double *pl, const double *pr, const FaceGeom<double> &g, double *flux, double &sig)
{
  return riemann3<DIR>(false, pl, pr, g, flux, sig);
}
template <int DIR, bool MIX>
__device__ __forceinline__ void hlle3(const double *pl, const double *pr, const FaceGeom<double> &g, double *flux, double &sig)
{
  riemann3<DIR, MIX>(true, pl, pr, g, flux, sig);
}

// Face geometry of direction d on row (i, j): area[d], scale[1+d][d], gcov[1+d][0..2].
template <int DIR>
__device__ __forceinline__ FaceGeom<double> face_geom3(const Grid3 &g, int ij)
{
  FaceGeom<double> f;
  f.area = geo3(g, G3_A0 + DIR, ij);
  f.scale = geo3(g, G3_SCALE + 3 * (1 + DIR) + DIR, ij);
  f.g0 = geo3(g, G3_GCOV + 3 * (1 + DIR) + 0, ij);
  f.g1 = geo3(g, G3_GCOV + 3 * (1 + DIR) + 1, ij);
  f.g2 = geo3(g, G3_GCOV + 3 * (1 + DIR) + 2, ij);
  return f;
}

// Right face value of pencil zone 1 and left face value of pencil zone 2 (interp() on a
// 4-zone pencil, reconstruct.c:225-279), reconstruction columns c1, c2 of table rc.
__device__ __forceinline__ void recon_face(int order, const double pen[4][7], const double *rc, int64_t stride,
                                           int64_t c1, int64_t c2, double *pl, double *pr)
{
  const RcView<double, true> g1{rc + c1, stride}, g2{rc + c2, stride};
  recon_vars<7>(order, g1, [&](int v, int q) { return pen[q][v]; }, [&](int v, double, double hi) { pl[v] = hi; });
  recon_vars<7>(order, g2, [&](int v, int q) { return pen[1 + q][v]; }, [&](int v, double lo, double) { pr[v] = lo; });
}

// Mixed precision (MIX): the same pencils, para_recon in FP32 difference form with the
// FP32 weights of the zone (face values a + da formed in FP64), HLLC with FP32 wave speeds
// and star-state increments and an FP64 upwind flux.  Faces the FP32 solver declines
// (ill-conditioned, MIX_COND_MAX) or whose Gamma slot is not the constant Gamma (the
// restricted radial entries) are re-solved in FP64 from the pencil; HLLE faces (next to
// a shock) take the FP64 solver on the mixed face states.
template <int DIR>
__device__ __noinline__ int face_fp64_3d(int order, const double *pen, const double *rc, int64_t stride, int64_t c1,
                                         int64_t c2, FaceGeom<double> fg, double *fl, double *ss)
{
  double p[4][7], pl[7], pr[7];
  for (int q = 0; q < 28; q++) p[q / 7][q % 7] = pen[q];
  recon_face(order, p, rc, stride, c1, c2, pl, pr);
  return hllc3<DIR>(pl, pr, fg, fl, *ss);
}

// Flag of zone (i, jj, kc) as transverse_shock reads it at this point of the serial loop.
template <int STAGE>
__device__ __forceinline__ bool flag_shock(const Grid3 &g, int i, int jj, int kc, const unsigned char *own,
                                           const unsigned char *all0)
{
  if (jj < 0 || jj >= nj_of(g, i)) return true;
  if (kc < 0 || kc >= nk_of(g, i, jj)) return true;
  const int64_t c = __ldg(g.cell + rowi(g, i, jj)) + kc;
  return own[c] != 0 || (STAGE == 1 && all0[c] != 0);
}

// Direction-0 faces: face (i, j, k) is the lower radial face of zone (i, j, k), i in [0, n1].
// A work item is a run of up to RUN0 consecutive radial faces i0 .. i0+ni-1 of one (j, k)
// column whose face rows share their theta and phi resolution (djs(i), dks(i, j)), so
// every pencil entry (radial row ii at that resolution) is the same for all faces of the
// run: each thread walks outwards through its column with a ring of pencil entries in
// shared memory, loads one new entry and reconstructs one zone per face (zone i's left
// face value for face i, its right face value kept for face i+1), where the reference's
// interp() builds a 4-zone pencil and reconstructs two zones per face.  The values are
// the same; only their reuse differs.
//
// Work list: a run is nr faces r0 .. r0+nr-1 of the fixed row `row` (the theta row j for
// direction 0, the radial row i for direction 1) in every phi column of the face row.  The
// columns of all runs, one per thread, stand one after the other in one line of lanes
// (runs of equal length together): column k of a run is lane l0 + k, CTA b takes lanes
// 128 b .. 128 b + 127, and first[b] is the run of its first lane.  Rows have 4 phi zones at
// the poles and 1 on the 2-D grid, so a CTA per row left most threads without work: 1.4
// active threads per warp instruction on a 2-D 400 x 256 grid (0.75 + 0.83 ms for the two
// kernels of a stage there).
struct Run3 { int r0, nr, row, l0; };
constexpr int RUN0 = 16;          // default of mdg_launch_config::run_length

// Direction-2 faces: up to T2 faces k0 .. k0+cnt-1 of row (i, j) on lanes l0 .. l0+cnt+1 of
// a CTA, the n-th segment of that CTA (n < SEG2_MAX).
struct Seg2 { int i, j, k0, cnt, l0, n; };
constexpr int SEG2_MAX = 18;      // most segments of a CTA (whole rows have at least 5 faces, 7 lanes)

// Which of a CTA's consecutive items (rows, runs, segments; at least one lane each) this
// thread's lane belongs to: start(q) is the first lane, relative to the CTA's, of its q-th
// item after the one its first lane belongs to (NT3 where there is none).
template <typename F>
__device__ __forceinline__ int item_of_lane(int *sbeg, F start)
{
  const int t = (int)threadIdx.x;
  sbeg[t] = start(1 + t);
  __syncthreads();
  int lo = 0;   // items after the first that start at or before this lane (at most NT3-1)
#pragma unroll
  for (int s = NT3 / 2; s > 0; s >>= 1)
    if (sbeg[lo + s - 1] <= t) lo += s;
  return lo;
}

// Thread of a zone kernel: the interior row (index into prow and rowcell) of zone c; CTA b
// takes the zones 128 b .. 128 b + 127 in zone order.
__device__ __forceinline__ int zone_row(const Grid3 &g, int *sbeg)
{
  const int64_t c0 = (int64_t)blockIdx.x * NT3;
  const int r0 = __ldg(g.row0 + blockIdx.x);
  return r0 + item_of_lane(sbeg, [&](int q) {
    const int64_t d = (r0 + q < g.nrow) ? __ldg(g.rowcell + r0 + q) - c0 : (int64_t)NT3;
    return d < NT3 ? (int)d : NT3;
  });
}

// Thread of a run kernel: its run.
__device__ __forceinline__ Run3 lane_run(const Run3 *__restrict__ runs, int nrun, const int *__restrict__ first, int *sbeg)
{
  const int r0 = __ldg(first + blockIdx.x), b0 = (int)blockIdx.x * NT3;
  const int q = item_of_lane(sbeg, [&](int k) {
    const int d = (r0 + k < nrun) ? runs[r0 + k].l0 - b0 : NT3;
    return d < NT3 ? d : NT3;
  });
  return runs[r0 + q];
}

// The RK stage is a run-time argument here (not a template argument as in the other
// face kernels): both stages then run the same code, which measured faster for stage 1
// than its own specialisation.
template <bool MIX, bool SMALL>
__global__ void __launch_bounds__(NT3, f3_minb(MIX, SMALL)) face0_kernel(const ProbDev *__restrict__ probs, ProbTime *__restrict__ times,
                                                     Grid3 g, const Run3 *__restrict__ runs, int nrun,
                                                     const int *__restrict__ first, int nlane, StateSoA s,
                                                     double *__restrict__ flux, unsigned char *__restrict__ own,
                                                     unsigned char *__restrict__ all0, int stage)
{
  // ring of pencil entries (radial rows i-1 .. i+1; i-2 as well for the FP64 re-solve of
  // the mixed sweep) and the right face values of the previous zone, [slot][var][thread]
  constexpr int NS = MIX ? 4 : 3;
  __shared__ double win[NS][7][NT3];
  __shared__ double arb[7][NT3];
  __shared__ double sred[32];
  __shared__ int sbeg[NT3];
  if (times[0].done) return;
  const ProbDev &P = probs[0];
  const int tid = (int)threadIdx.x, lane = (int)blockIdx.x * NT3 + tid;
  const Run3 t = lane_run(runs, nrun, first, sbeg);
  double lmin = 1.0e300;
  if (lane < nlane) {
    const int i0 = t.r0, j = t.row, k = lane - t.l0;
    const int64_t rcs = g.n1 + 2 * NG;
    auto slot = [&](int ii) { return (ii - i0 + 2) % NS; };
    // The rows of the run stand at the faces' resolution: each is its own pencil entry and is read
    // directly.  Rows of other levels, ghost rows and zones with a -0 take the general entry,
    // whose index tables, integer divisions and dependent loads every entry went through before:
    // 384 x 128 x 256 blast, plain FP64 7.10 -> 6.84 ms per step (6.62 with riemann3), mixed 5.46 -> 5.26 ms.  On
    // small grids, whose runs are a face or two, the rows beside the run are tested as well
    // (2-D 400 x 256 mixed 170 -> 162 us; on the large grid the test cost 0.3 ms).  zone_of runs
    // one row ahead of the loads, so that the row tables' latency is not waited for.
    const int nj_face = nj_of(g, i0), nk_face = nk_of(g, i0, j);
    auto zone_of = [&](int ii) -> int64_t {
      if (!SMALL) return (ii >= i0 && ii < i0 + t.nr && ii < g.n1) ? __ldg(g.cell + rowi(g, ii, j)) + k : -1;
      if (ii < 0 || ii >= g.n1 || nj_of(g, ii) != nj_face) return -1;
      const int r = rowi(g, ii, j);
      return __ldg(g.nk + r) == nk_face ? __ldg(g.cell + r) + k : -1;
    };
    int64_t zone = zone_of(i0 - 2);
    auto entry = [&](int ii, int64_t c) {
      double w[7];
      if (c < 0 || load7_zone(P, s, c, w)) pencil0(g, P, s, i0, j, k, ii, w);
#pragma unroll
      for (int v = 0; v < 7; v++) win[slot(ii)][v][tid] = w[v];
    };
#pragma unroll 1
    for (int ii = i0 - 2; ii <= i0; ii++) {
      entry(ii, zone);
      zone = zone_of(ii + 1);
    }
    {
      // right face values of zone i0-1
      const int sm = slot(i0 - 2), s0 = slot(i0 - 1), sp = slot(i0);
      if (MIX) {
        const MixW w = load_mixw(g.mx0 + i0 - 1 + NG, rcs);
#pragma unroll
        for (int v = 0; v < 7; v++) {
          const double a = win[s0][v][tid];
          float dl, dr;
          mixed_recon((float)(a - win[sm][v][tid]), (float)(win[sp][v][tid] - a), w, dl, dr);
          arb[v][tid] = a + (double)dr;
        }
      } else {
        const RcView<double, true> gz{g.rc0 + i0 - 1 + NG, rcs};
        recon_vars<7>(P.interp_order, gz, [&](int v, int q) { return win[q == 0 ? sm : q == 1 ? s0 : sp][v][tid]; },
                      [&](int v, double, double hi) { arb[v][tid] = hi; });
      }
    }
#pragma unroll 1
    for (int i = i0; i < i0 + t.nr; i++) {
      entry(i + 1, zone);
      zone = zone_of(i + 2);
      double pl[7], pr[7];
      const int sm = slot(i - 1), s0 = slot(i), sp = slot(i + 1);
      if (MIX) {
        const MixW w = load_mixw(g.mx0 + i + NG, rcs);
#pragma unroll
        for (int v = 0; v < 7; v++) {
          pl[v] = arb[v][tid];
          const double a = win[s0][v][tid];
          float dl, dr;
          mixed_recon((float)(a - win[sm][v][tid]), (float)(win[sp][v][tid] - a), w, dl, dr);
          pr[v] = a + (double)dl;
          arb[v][tid] = a + (double)dr;
        }
      } else {
        const RcView<double, true> gz{g.rc0 + i + NG, rcs};
        recon_vars<7>(P.interp_order, gz, [&](int v, int q) { return win[q == 0 ? sm : q == 1 ? s0 : sp][v][tid]; },
                      [&](int v, double lo, double hi) { pl[v] = arb[v][tid]; pr[v] = lo; arb[v][tid] = hi; });
      }
      const int ij = rowi(g, i, j);
      const FaceGeom<double> fg = face_geom3<0>(g, ij);
      double fl[NPRIM], ss;
      int isshock = -1;
      if (!MIX) {
        isshock = riemann3<0>(false, pl, pr, fg, fl, ss);
      } else {
        if (pl[6] == P.gam && pr[6] == P.gam) {
          float sig;
          int sh;
          if (riemann_hllc_mixed<0>(pl, pr, fg, gam_const<float>((float)P.gam), fl, sig, sh)) {
            ss = (double)sig;
            isshock = sh;
          }
        }
        if (isshock < 0) {
          double pen[28];
#pragma unroll
          for (int q = 0; q < 28; q++) pen[q] = win[slot(i - 2 + q / 7)][q % 7][tid];
          isshock = face_fp64_3d<0>(P.interp_order, pen, g.rc0, rcs, i - 1 + NG, i + NG, fg, fl, &ss);
        }
      }
      const int64_t f = __ldg(g.f0 + ij) + k;
#pragma unroll
      for (int v = 0; v < NPRIM; v++) flux[v * g.nf0 + f] = fl[v];
      if (i < g.n1) own[__ldg(g.cell + ij) + k] = (unsigned char)isshock;
      if (stage == 0 && isshock) {
        // shock marks of the zone and of the two zones inside it (step.c:1196-1204)
        if (i < g.n1) all0[__ldg(g.cell + ij) + k] = 1;
        for (int d = 1; d <= 2; d++) {
          const int im = i - d;
          if (im < 0) break;
          const int jm = j * djs(g, i) / djs(g, im);
          const int km = k * dks(g, i, j) / dks(g, im, jm);
          all0[__ldg(g.cell + rowi(g, im, jm)) + km] = 1;
        }
      }
      lmin = tmin(lmin, g.dx0 / fabs(ss));
    }
  }
  block_min_to(lmin, &times[0].minacc, sred);
}

// Direction-1 faces: sub-face kk of face row (i, j), j in [0, nj(i)] (step.c:1212-1265).
// As for direction 0, a work item is a run of up to RUN0 consecutive faces j0 .. j0+nj-1
// of radial row i and sub-face column kk whose face rows share their phi resolution
// mn = min(dks(i, j), dks(i, j-1)) (every pencil entry, theta row jj at that resolution,
// is then the same for all faces of the run); a thread walks northwards through its
// column, one new entry and one zone reconstruction per face.  Run3 fields here:
// r0 = j0, nr = faces, row = i.
template <bool MIX, bool SMALL>
__global__ void __launch_bounds__(NT3, f3_minb(MIX, SMALL)) face1_kernel(const ProbDev *__restrict__ probs, ProbTime *__restrict__ times,
                                                     Grid3 g, const Run3 *__restrict__ runs, int nrun,
                                                     const int *__restrict__ first, int nlane, StateSoA s,
                                                     double *__restrict__ flux, const unsigned char *__restrict__ own,
                                                     const unsigned char *__restrict__ all0, int stage)
{
  constexpr int NS = MIX ? 4 : 3;
  __shared__ double win[NS][7][NT3];
  __shared__ double arb[7][NT3];
  __shared__ double sred[32];
  __shared__ int sbeg[NT3];
  if (times[0].done) return;
  const ProbDev &P = probs[0];
  const int tid = (int)threadIdx.x, lane = (int)blockIdx.x * NT3 + tid;
  const Run3 t = lane_run(runs, nrun, first, sbeg);
  double lmin = 1.0e300;
  if (lane < nlane) {
    const int j0 = t.r0, i = t.row, kk = lane - t.l0;
    const int64_t cs = g.cols1;
    const int64_t base = g.rc1_base[ilog2(djs(g, i))] + NG;
    auto slot = [&](int jj) { return (jj - j0 + 2) % NS; };
    // As in face0_kernel: an interior theta row at the faces' phi resolution is its own entry.
    const int row_i = rowi(g, i, 0), nj_i = nj_of(g, i);
    const int nk_face = max(nk_of(g, i, j0), nk_of(g, i, j0 - 1));
    auto zone_of = [&](int jj) -> int64_t {
      return (jj >= 0 && jj < nj_i && __ldg(g.nk + row_i + jj) == nk_face) ? __ldg(g.cell + row_i + jj) + kk : -1;
    };
    int64_t zone = zone_of(j0 - 2);
    auto entry = [&](int jj, int64_t c) {
      double w[7];
      if (c < 0) pencil1(g, P, s, i, j0, kk, jj, w);
      else load7_zone(P, s, c, w);
#pragma unroll
      for (int v = 0; v < 7; v++) win[slot(jj)][v][tid] = w[v];
    };
#pragma unroll 1
    for (int jj = j0 - 2; jj <= j0; jj++) {
      const int64_t c = zone;
      zone = zone_of(jj + 1);
      entry(jj, c);
    }
    {
      // right face values of zone j0-1
      const int sm = slot(j0 - 2), s0 = slot(j0 - 1), sp = slot(j0);
      if (MIX) {
        const MixW w = load_mixw(g.mx1 + base + j0 - 1, cs);
#pragma unroll
        for (int v = 0; v < 7; v++) {
          const double a = win[s0][v][tid];
          float dl, dr;
          mixed_recon((float)(a - win[sm][v][tid]), (float)(win[sp][v][tid] - a), w, dl, dr);
          arb[v][tid] = a + (double)dr;
        }
      } else {
        const RcView<double, true> gz{g.rc1 + base + j0 - 1, cs};
        recon_vars<7>(P.interp_order, gz, [&](int v, int q) { return win[q == 0 ? sm : q == 1 ? s0 : sp][v][tid]; },
                      [&](int v, double, double hi) { arb[v][tid] = hi; });
      }
    }
#pragma unroll 1
    for (int j = j0; j < j0 + t.nr; j++) {
      entry(j + 1, zone);
      zone = zone_of(j + 2);
      double pl[7], pr[7];
      const int sm = slot(j - 1), s0 = slot(j), sp = slot(j + 1);
      if (MIX) {
        const MixW w = load_mixw(g.mx1 + base + j, cs);
#pragma unroll
        for (int v = 0; v < 7; v++) {
          pl[v] = arb[v][tid];
          const double a = win[s0][v][tid];
          float dl, dr;
          mixed_recon((float)(a - win[sm][v][tid]), (float)(win[sp][v][tid] - a), w, dl, dr);
          pr[v] = a + (double)dl;
          arb[v][tid] = a + (double)dr;
        }
      } else {
        const RcView<double, true> gz{g.rc1 + base + j, cs};
        recon_vars<7>(P.interp_order, gz, [&](int v, int q) { return win[q == 0 ? sm : q == 1 ? s0 : sp][v][tid]; },
                      [&](int v, double lo, double hi) { pl[v] = arb[v][tid]; pr[v] = lo; arb[v][tid] = hi; });
      }
      // zone k of row j that owns the sub-face, and the transverse_shock test of zone k
      const int dkj = dks(g, i, j), dkjm = dks(g, i, j - 1);
      const int mn = dkj < dkjm ? dkj : dkjm;
      const int k = kk / (dkj / mn);
      const int nkm = dkj / dkjm;
      bool hlle = (stage == 0) ? flag_shock<0>(g, i, j, k, own, all0) : flag_shock<1>(g, i, j, k, own, all0);
      for (int q = k * nkm; q < k * nkm + nkm; q++)
        hlle = hlle || ((stage == 0) ? flag_shock<0>(g, i, j - 1, q, own, all0) : flag_shock<1>(g, i, j - 1, q, own, all0));
      const int ij = rowi(g, i, j);
      const FaceGeom<double> fg = face_geom3<1>(g, ij);
      double fl[NPRIM], ss;
      if (!MIX) {
        riemann3<1>(hlle, pl, pr, fg, fl, ss);
      } else if (hlle) {
        hlle3<1, MIX>(pl, pr, fg, fl, ss);
      } else {
        bool done = false;
        if (pl[6] == P.gam && pr[6] == P.gam) {
          float sig;
          int sh;
          if (riemann_hllc_mixed<1>(pl, pr, fg, gam_const<float>((float)P.gam), fl, sig, sh)) {
            ss = (double)sig;
            done = true;
          }
        }
        if (!done) {
          double pen[28];
#pragma unroll
          for (int q = 0; q < 28; q++) pen[q] = win[slot(j - 2 + q / 7)][q % 7][tid];
          face_fp64_3d<1>(P.interp_order, pen, g.rc1, cs, base + j - 1, base + j, fg, fl, &ss);
        }
      }
      const int64_t f = __ldg(g.f1 + ij) + kk;
#pragma unroll
      for (int v = 0; v < NPRIM; v++) flux[v * g.nf1 + f] = fl[v];
      lmin = tmin(lmin, djs(g, i) * g.dx1 / fabs(ss));
    }
  }
  block_min_to(lmin, &times[0].minacc, sred);
}

// Direction-2 faces: face k in [0, nk] of row (i, j) (step.c:1267-1425), with the
// polar-axis fix on the last theta row.  A CTA takes segments of consecutive faces of one
// row each (Seg2; short rows share a CTA, a long one is cut): per segment it stages the
// zones they read in shared memory (each zone loaded once) and reconstructs every zone
// once (the reference reconstructs each zone for both of its faces), then a thread solves
// one face.  With one row per CTA the 128 x 64 x 128 grid ran 13274 CTAs at 20 active
// threads per warp instruction (0.36 ms a stage, plain FP64).
constexpr int T2 = NT3 - 2;
template <int STAGE, bool MIX, bool SMALL>
__global__ void __launch_bounds__(NT3, f3_minb(MIX, SMALL)) face2_kernel(const ProbDev *__restrict__ probs, ProbTime *__restrict__ times,
                                                     Grid3 g, const Seg2 *__restrict__ segs, int nseg,
                                                     const int *__restrict__ first, StateSoA s,
                                                     double *__restrict__ flux, const unsigned char *__restrict__ own,
                                                     const unsigned char *__restrict__ all0)
{
  __shared__ double sv_[7][NT3 + 2 * SEG2_MAX];   // zones k0-2 .. k0+cnt+1 of each segment
  __shared__ double sal_[7][NT3];                 // left / right face values of zones k0-1 .. k0+cnt
  __shared__ double sar_[7][NT3];
  __shared__ double sred[32];
  __shared__ int sbeg[NT3];
  if (times[0].done) return;
  const ProbDev &P = probs[0];
  const int s0 = __ldg(first + blockIdx.x);
  const Seg2 tl = segs[s0 + item_of_lane(sbeg, [&](int q) {
    return (q < SEG2_MAX && s0 + q < nseg && segs[s0 + q].n == q) ? segs[s0 + q].l0 : NT3;
  })];
  const int i = tl.i, j = tl.j, k0 = tl.k0, cnt = tl.cnt;
  const int t = (int)threadIdx.x - tl.l0;   // lane within the segment; past cnt+1: no work
  // this segment's part of the shared arrays, indexed by t
  double (*sv)[NT3 + 2 * SEG2_MAX] = reinterpret_cast<double(*)[NT3 + 2 * SEG2_MAX]>(&sv_[0][tl.l0 + 2 * tl.n]);
  double (*sal)[NT3] = reinterpret_cast<double(*)[NT3]>(&sal_[0][tl.l0]);
  double (*sar)[NT3] = reinterpret_cast<double(*)[NT3]>(&sar_[0][tl.l0]);
  const int ij = rowi(g, i, j);
  const int dk = dks(g, i, j);
  const int64_t base = g.rc2_base[ilog2(dk)] + NG;
  const bool pole = (j == nj_of(g, i) - 1);
  if (t < cnt + 2) {
    double w[7];
    load7(g, P, s, i, j, k0 - 1 + t, w);
#pragma unroll
    for (int v = 0; v < 7; v++) sv[v][t + 1] = w[v];
    if (t == 0 || t == cnt + 1) {
      const int e = t == 0 ? 0 : cnt + 3;
      load7(g, P, s, i, j, k0 - 2 + e, w);
#pragma unroll
      for (int v = 0; v < 7; v++) sv[v][e] = w[v];
    }
  }
  __syncthreads();
  if (!pole && t < cnt + 2) {
    // zone k0-1+t from the staged neighbours (interp() on its 3-zone stencil)
    if (MIX) {
      const MixW w = load_mixw(g.mx2 + base + k0 - 1 + t, g.cols2);
#pragma unroll
      for (int v = 0; v < 7; v++) {
        float dl, dr;
        const double a = sv[v][t + 1];
        mixed_recon((float)(a - sv[v][t]), (float)(sv[v][t + 2] - a), w, dl, dr);
        sal[v][t] = a + (double)dl;
        sar[v][t] = a + (double)dr;
      }
    } else {
      const RcView<double, true> gz{g.rc2 + base + k0 - 1 + t, g.cols2};
      recon_vars<7>(P.interp_order, gz, [&](int v, int q) { return sv[v][t + q]; },
                    [&](int v, double lo, double hi) { sal[v][t] = lo; sar[v][t] = hi; });
    }
  }
  __syncthreads();
  double lmin = 1.0e300;
  if (t < cnt) {
    const int k = k0 + t;
    double pl[7], pr[7];
    if (pole) {
      // polar-axis fix: zone values, velocity rotated at the shared phi face
      const int64_t b1 = g.rc1_base[ilog2(djs(g, i))] + NG + j;
      const double sth = __ldg(g.sth + b1), cth = __ldg(g.cth + b1);
      double s0[3], s3[3];
#pragma unroll
      for (int m = 0; m < 3; m++) {
        s0[m] = geo3(g, G3_SCALE + m, ij);
        s3[m] = geo3(g, G3_SCALE + 9 + m, ij);
      }
      const double sphf = __ldg(g.sphl + base + k), cphf = __ldg(g.cphl + base + k);
      for (int side = 0; side < 2; side++) {
        const int kt = k - 1 + side;
        double w[7];
#pragma unroll
        for (int v = 0; v < 7; v++) w[v] = sv[v][t + 1 + side];
        const double sph = __ldg(g.sphc + base + kt), cph = __ldg(g.cphc + base + kt);
        double lam[3][3] = {{sth * cph, cth * cph, -sph}, {sth * sph, cth * sph, cph}, {cth, -sth, 0.0}};
        double v[3];
        for (int l = 0; l < 3; l++) {
          v[l] = 0.0;
          for (int m = 0; m < 3; m++) v[l] += lam[l][m] * w[U1 + m] * s0[m];
        }
        double lf[3][3] = {{sth * cphf, cth * cphf, -sphf}, {sth * sphf, cth * sphf, cphf}, {cth, -sth, 0.0}};
        double *o = side ? pr : pl;
#pragma unroll
        for (int q = 0; q < 7; q++) o[q] = w[q];
        for (int l = 0; l < 3; l++) {
          o[U1 + l] = 0.0;
          for (int m = 0; m < 3; m++) o[U1 + l] += lf[m][l] * v[m] / s3[l];
        }
      }
    } else {
#pragma unroll
      for (int v = 0; v < 7; v++) {
        pl[v] = sar[v][t];
        pr[v] = sal[v][t + 1];
      }
    }
    const bool hlle = flag_shock<STAGE>(g, i, j, k, own, all0) || flag_shock<STAGE>(g, i, j, k - 1, own, all0);
    const FaceGeom<double> fg = face_geom3<2>(g, ij);
    double fl[NPRIM], ss;
    if (!MIX) {
      riemann3<2>(hlle, pl, pr, fg, fl, ss);
    } else if (hlle) {
      hlle3<2, MIX>(pl, pr, fg, fl, ss);
    } else {
      float sig;
      int isshock;
      if (pl[6] == P.gam && pr[6] == P.gam &&
          riemann_hllc_mixed<2>(pl, pr, fg, gam_const<float>((float)P.gam), fl, sig, isshock)) {
        ss = (double)sig;
      } else if (pole) {
        hllc3<2>(pl, pr, fg, fl, ss);
      } else {
        double pen[4][7];
#pragma unroll
        for (int q = 0; q < 28; q++) pen[q / 7][q % 7] = sv[q % 7][t + q / 7];
        face_fp64_3d<2>(P.interp_order, &pen[0][0], g.rc2, g.cols2, base + k - 1, base + k, fg, fl, &ss);
      }
    }
    const int64_t f = __ldg(g.f2 + ij) + k;
#pragma unroll
    for (int v = 0; v < NPRIM; v++) flux[v * g.nf2 + f] = fl[v];
    lmin = dk * g.dx2 / fabs(ss);
  }
  block_min_to(lmin, &times[0].minacc, sred);
}

// The face launches of one RK stage, plain FP64 (mdg_sweep3d.cu) or mixed
// (mdg_sweep3d_mixed.cu): work lists, fluxes and shock bits as Sweep3 holds them.
struct FaceLaunch3 {
  int nt[3];                        // CTAs of the three kernels
  bool small[3];                    // at most F3MINB_SMALL CTAs per SM
  const Run3 *runs[2];
  const int *first[3];
  int nrun[2], nlane[2], nseg;
  const Seg2 *segs;
  double *F[3];
  unsigned char *own, *all0;
};
template <int STAGE, bool MIX>
inline void launch_faces3(const FaceLaunch3 &f, const ProbDev *probs, ProbTime *times, const Grid3 &g, StateSoA s,
                          cudaStream_t st)
{
  auto k0 = f.small[0] ? face0_kernel<MIX, true> : face0_kernel<MIX, false>;
  auto k1 = f.small[1] ? face1_kernel<MIX, true> : face1_kernel<MIX, false>;
  auto k2 = f.small[2] ? face2_kernel<STAGE, MIX, true> : face2_kernel<STAGE, MIX, false>;
  k0<<<f.nt[0], NT3, 0, st>>>(probs, times, g, f.runs[0], f.nrun[0], f.first[0], f.nlane[0], s, f.F[0], f.own, f.all0,
                              STAGE);
  k1<<<f.nt[1], NT3, 0, st>>>(probs, times, g, f.runs[1], f.nrun[1], f.first[1], f.nlane[1], s, f.F[1], f.own, f.all0,
                              STAGE);
  if (f.nt[2] > 0)
    k2<<<f.nt[2], NT3, 0, st>>>(probs, times, g, f.segs, f.nseg, f.first[2], s, f.F[2], f.own, f.all0);
}
void launch_faces3_mixed(int stage, const FaceLaunch3 &f, const ProbDev *probs, ProbTime *times, const Grid3 &g,
                         StateSoA s, cudaStream_t st);

}  // namespace mdg
