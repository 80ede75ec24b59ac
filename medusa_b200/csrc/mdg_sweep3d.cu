// 3-D (and 2-D spherical) dendritic sweep: the zone update, the work lists and the launches.  The
// face kernels of both precisions are in mdg_sweep3d.cuh; the plain FP64 ones are built here.
#include "mdg_sweep3d.cuh"
#include <algorithm>
#include <string>
#include <vector>

namespace mdg {

// monopole_gravity_start (gravity.c:238-246): mass vol*rho of radial shell i, summed over
// its zones in zone order (one thread per shell, the reference's serial order).
__global__ void shell_mass3_kernel(const ProbTime *__restrict__ times, Grid3 g, StateSoA s)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n1 || times[0].done) return;
  double ms = 0.0;
  for (int j = 0; j < nj_of(g, i); j++) {
    const int ij = rowi(g, i, j);
    const double vol = geo3(g, G3_VOL, ij);
    const int64_t c0 = __ldg(g.cell + ij);
    const int nk = __ldg(g.nk + ij);
#pragma unroll 8
    for (int k = 0; k < nk; k++) ms += vol * s.v[RHO][c0 + k];
  }
  g.gmono[i] = ms;
}

// monopole_gravity_finish (gravity.c:300-319, GR_MONOPOLE=FALSE): enclosed mass at the
// radial edges, g = -G mr / r^2 dr/dx there, interpolated to the zone centroids (in place
// over the shell masses).
__global__ void monopole_profile3_kernel(const ProbTime *__restrict__ times, Grid3 g)
{
  if (threadIdx.x != 0 || times[0].done) return;
  const int64_t rcs = g.n1 + 2 * NG;
  double mr = 0.0, gl = 0.0;
  for (int ii = 0; ii < g.n1; ii++) {
    mr = mr + g.gmono[ii];
    const double gr = -GNEWT * mr / __ldg(g.medge + ii + 1) * __ldg(g.medge + g.n1 + 1 + ii + 1);
    g.gmono[ii] = monopole_centroid(gl, gr, g.x0 + ii * g.dx0, g.dx0, __ldg(g.rc0 + RC_B0 * rcs + ii + NG),
                                    __ldg(g.rc0 + RC_G0 * rcs + ii + NG));
    gl = gr;
  }
}

// push() for zone (i, j, k) (step.c:327-478) with the dendritic flux fan-in, the
// geometric sources of the stage state (rad_fluid.c:164-192, fluid.c:56-73), fixed or
// monopole gravity and, in the
// second stage, the zone terms of the next estimate_dt (step.c:177-187).
template <int STAGE>
__global__ void __launch_bounds__(NT3, MDG_P3MINB) push3_kernel(const ProbDev *__restrict__ probs, ProbTime *__restrict__ times,
                                                     Grid3 g, StateSoA sst,
                                                     StateSoA sn, StateSoA out, const double *__restrict__ F0,
                                                     const double *__restrict__ F1, const double *__restrict__ F2)
{
  __shared__ double sred[32];
  __shared__ int sbeg[NT3];
  if (times[0].done) return;
  const ProbDev &P = probs[0];
  const double dt = times[0].dt;
  const int64_t c = (int64_t)blockIdx.x * NT3 + threadIdx.x;
  const int row = zone_row(g, sbeg);
  double lmin = 1.0e300;
  if (c < g.ncell) {
    const PushRow3 &pr = g.prow[row];
    const int i = pr.i, j = pr.j, ij = pr.ij, k = (int)(c - __ldg(g.rowcell + row));
    double ph[NPRIM], pn[NPRIM], u[NPRIM], uh[NPRIM], src[NPRIM], divF[NPRIM], pf[NPRIM];
#pragma unroll
    for (int v = 0; v < NPRIM; v++) ph[v] = sst.v[v][c];
    if (STAGE == 0) {
#pragma unroll
      for (int v = 0; v < NPRIM; v++) pn[v] = ph[v];
    } else {
#pragma unroll
      for (int v = 0; v < NPRIM; v++) pn[v] = sn.v[v][c];
    }
    const double g0 = geo3(g, G3_GCOV + 0, ij), g1 = geo3(g, G3_GCOV + 1, ij), g2 = geo3(g, G3_GCOV + 2, ij);
    const double press = eos_press(P.eos, P.gam, P.Kpoly, ph[RHO], ph[UU]);
    {
      // p_to_geom_src: src[U1+m] = sum_l sum_n T[l][n] conn[l][m][n] over the non-zero conn
      const double vcov[3] = {g0 * ph[U1], g1 * ph[U2], g2 * ph[U3]};
      double T[3][3];
#pragma unroll
      for (int l = 0; l < 3; l++) {
#pragma unroll
        for (int m = 0; m < 3; m++) T[l][m] = ph[RHO] * ph[U1 + m] * vcov[l];
        T[l][l] += press;
      }
      double s0 = 0.0, s1 = 0.0, s2 = 0.0;
      s0 += T[0][0] * geo3(g, G3_C000, ij);
      s0 += T[1][1] * geo3(g, G3_C101, ij);
      s0 += T[2][2] * geo3(g, G3_C202, ij);
      s1 += T[0][1] * geo3(g, G3_C011, ij);
      s1 += T[1][0] * geo3(g, G3_C110, ij);
      s1 += T[1][1] * geo3(g, G3_C111, ij);
      s1 += T[2][2] * geo3(g, G3_C212, ij);
      s2 += T[0][2] * geo3(g, G3_C022, ij);
      s2 += T[1][2] * geo3(g, G3_C122, ij);
      s2 += T[2][0] * geo3(g, G3_C220, ij);
      s2 += T[2][1] * geo3(g, G3_C221, ij);
      src[RHO] = 0.0; src[UU] = 0.0; src[U1] = s0; src[U2] = s1; src[U3] = s2;
    }
    // GRAV=FIXED_GRAV (gravity.c:38-64): the constant contravariant acceleration, lowered
    // with the zone's metric, on the momenta of the grid's directions and the energy
    if (P.grav_on) add_fixed_gravity(ph, P.grav, g0, g1, g2, g.ndim, src);
    if (g.mono) {
      // monopole gravity (gravity.c:373-401): mass flux density on the outer faces of the
      // zone (row i+1, the fan-in below) and on its inner face
      const int dji = djs(g, i), djo = djs(g, i + 1);
      const int jp = j * dji / djo, njp = dji / djo, dkij = dks(g, i, j);
      double vr = 0.0, area = 0.0;
      for (int jj = jp; jj < jp + njp; jj++) {
        const int nkp = dkij / dks(g, i + 1, jj);
        const int ijo = rowi(g, i + 1, jj);
        const int64_t fb = __ldg(g.f0 + ijo);
        const double ao = geo3(g, G3_A0, ijo);
        for (int kk = k * nkp; kk < k * nkp + nkp; kk++) {
          vr += F0[RHO * g.nf0 + fb + kk];
          area += ao + 1.0e-16;
        }
      }
      vr /= area;
      const double vl = F0[RHO * g.nf0 + __ldg(g.f0 + ij) + k] / (geo3(g, G3_A0, ij) + 1.0e-16);
      const int64_t rcs = g.n1 + 2 * NG;
      add_monopole_gravity(ph[RHO], g.gmono[i], vl, vr, g.x0 + i * g.dx0, g.dx0, __ldg(g.rc0 + RC_B0 * rcs + i + NG),
                           __ldg(g.rc0 + RC_G0 * rcs + i + NG), src);
    }
    p_to_u(pn, u, g0, g1, g2);
    p_to_u(ph, uh, g0, g1, g2);
    lmin = dt_source_control(pn, u, src);
#pragma unroll
    for (int v = 0; v < NPRIM; v++) divF[v] = 0.0;
    // direction 0: outer face(s) on row i+1, inner face
    {
      const int nf0o = pr.nf0o;
      for (int q = 0; q < nf0o; q++) {
        const int nkp = pr.nkp[q];
        const int64_t fb = pr.f0o[q];
        for (int kk = k * nkp; kk < k * nkp + nkp; kk++) {
#pragma unroll
          for (int v = 0; v < NPRIM; v++) divF[v] += F0[v * g.nf0 + fb + kk];
        }
      }
      const int64_t fi = pr.f0i + k;
#pragma unroll
      for (int v = 0; v < NPRIM; v++) divF[v] -= F0[v * g.nf0 + fi];
    }
    // direction 1
    {
      const int64_t fo = pr.f1o, fin = pr.f1i;
      const int mo = pr.mo, mi = pr.mi;
      if (mo == 1) {
#pragma unroll
        for (int v = 0; v < NPRIM; v++) divF[v] += 0.5 * F1[v * g.nf1 + fo + k];
      } else if (mo == 2) {
#pragma unroll
        for (int v = 0; v < NPRIM; v++) divF[v] += F1[v * g.nf1 + fo + 2 * k] + F1[v * g.nf1 + fo + 2 * k + 1];
      } else {
#pragma unroll
        for (int v = 0; v < NPRIM; v++) divF[v] += F1[v * g.nf1 + fo + k];
      }
      if (mi == 1) {
#pragma unroll
        for (int v = 0; v < NPRIM; v++)
          divF[v] -= 0.5 * F1[v * g.nf1 + fin + 2 * k] + 0.5 * F1[v * g.nf1 + fin + 2 * k + 1];
      } else {
#pragma unroll
        for (int v = 0; v < NPRIM; v++) divF[v] -= F1[v * g.nf1 + fin + k];
      }
    }
    // direction 2
    if (g.ndim == 3) {
      const int64_t f2 = pr.f2 + k;
#pragma unroll
      for (int v = 0; v < NPRIM; v++) divF[v] += F2[v * g.nf2 + f2 + 1] - F2[v * g.nf2 + f2];
    }
    const double vol = geo3(g, G3_VOL, ij);
    const double pfact = STAGE ? 0.5 : 1.0, phfact = STAGE ? 0.5 : 0.0, ffact = STAGE ? 0.5 : 1.0;
    double dv[NPRIM];
    quotients<NPRIM>(divF, vol, dv);
#pragma unroll
    for (int v = 0; v < NPRIM; v++) {
      const double ddt = dv[v] - src[v];
      u[v] = pfact * u[v] + phfact * uh[v] - ffact * dt * ddt;
    }
    u_to_p(u, pf, geo3(g, G3_GCON + 0, ij), geo3(g, G3_GCON + 1, ij), geo3(g, G3_GCON + 2, ij), P.floors != 0,
           P.rho_floor, P.e_floor);
#pragma unroll
    for (int v = 0; v < NPRIM; v++) out.v[v][c] = pf[v];
    flag_nonfinite(pf, &times[0]);
    if (STAGE == 1) {
      // next estimate_dt: velocity of the new state, sound speed of the stage state
      const double cs = sqrt(P.gam * press / ph[RHO]);
      double local_dt = 0.0;
      local_dt += (fabs(pf[U1]) + cs / geo3(g, G3_SCALE + 0, ij)) / g.dx0;
      lmin = tmin(lmin, 1.0 / local_dt);
      local_dt += (fabs(pf[U2]) + cs / geo3(g, G3_SCALE + 1, ij)) / (g.dx1 * djs(g, i));
      lmin = tmin(lmin, 1.0 / local_dt);
      if (g.ndim == 3) {
        local_dt += (fabs(pf[U3]) + cs / geo3(g, G3_SCALE + 2, ij)) / (g.dx2 * dks(g, i, j));
        lmin = tmin(lmin, 1.0 / local_dt);
      }
    }
  }
  block_min_to(lmin, &times[0].minacc, sred);
}

// First estimate_dt of the problem (step.c:171-187, the EOS of the state itself).
__global__ void __launch_bounds__(NT3) estimate3_kernel(const ProbDev *__restrict__ probs,
                                                         ProbTime *__restrict__ times, Grid3 g, StateSoA s)
{
  __shared__ double sred[32];
  __shared__ int sbeg[NT3];
  const ProbDev &P = probs[0];
  const int64_t c = (int64_t)blockIdx.x * NT3 + threadIdx.x;
  const int row = zone_row(g, sbeg);
  double lmin = 1.0e300;
  if (c < g.ncell) {
    const PushRow3 &pr = g.prow[row];
    const int i = pr.i, j = pr.j, ij = pr.ij;
    const double rho = s.v[RHO][c], uu = s.v[UU][c];
    const double cs = sqrt(P.gam * eos_press(P.eos, P.gam, P.Kpoly, rho, uu) / rho);
    double local_dt = 0.0;
    local_dt += (fabs(s.v[U1][c]) + cs / geo3(g, G3_SCALE + 0, ij)) / g.dx0;
    lmin = tmin(lmin, 1.0 / local_dt);
    local_dt += (fabs(s.v[U2][c]) + cs / geo3(g, G3_SCALE + 1, ij)) / (g.dx1 * djs(g, i));
    lmin = tmin(lmin, 1.0 / local_dt);
    if (g.ndim == 3) {
      local_dt += (fabs(s.v[U3][c]) + cs / geo3(g, G3_SCALE + 2, ij)) / (g.dx2 * dks(g, i, j));
      lmin = tmin(lmin, 1.0 / local_dt);
    }
  }
  block_min_to(lmin, &times[0].minacc, sred);
}


// Mass and total energy (utils.c:2337-2361, 2581-2612) with compensated sums: one CTA,
// each thread over a fixed subset of the zone tiles, then the threads in order.
__device__ __forceinline__ void neumaier3(double &s, double &c, double x)
{
  const double t = s + x;
  if (fabs(s) >= fabs(x)) c += (s - t) + x;
  else c += (x - t) + s;
  s = t;
}

__global__ void __launch_bounds__(256) totals3_kernel(Grid3 g, const Tile3 *__restrict__ tiles, int ntiles,
                                                       StateSoA s, double *__restrict__ out)
{
  __shared__ double sh[4][256];
  const int t = threadIdx.x;
  double ms = 0.0, mc = 0.0, es = 0.0, ec = 0.0;
  for (int q = t; q < ntiles; q += blockDim.x) {
    const Tile3 tl = tiles[q];
    const int ij = rowi(g, tl.i, tl.j);
    const double vol = geo3(g, G3_VOL, ij);
    const double g0 = geo3(g, G3_GCOV + 0, ij), g1 = geo3(g, G3_GCOV + 1, ij), g2 = geo3(g, G3_GCOV + 2, ij);
    for (int k = tl.k0; k < tl.k0 + tl.cnt; k++) {
      const int64_t c = __ldg(g.cell + ij) + k;
      double p[NPRIM], u[NPRIM];
#pragma unroll
      for (int v = 0; v < NPRIM; v++) p[v] = s.v[v][c];
      p_to_u(p, u, g0, g1, g2);
      neumaier3(ms, mc, p[RHO] * vol);
      neumaier3(es, ec, u[UU] * vol);
    }
  }
  sh[0][t] = ms; sh[1][t] = mc; sh[2][t] = es; sh[3][t] = ec;
  __syncthreads();
  if (t == 0) {
    double S = 0.0, C = 0.0, E = 0.0, D = 0.0;
    for (int k = 0; k < (int)blockDim.x; k++) {
      neumaier3(S, C, sh[0][k]); C += sh[1][k];
      neumaier3(E, D, sh[2][k]); D += sh[3][k];
    }
    out[0] = S + C;
    out[1] = E + D;
  }
}

// ------------------------------------------------------------------------ host driver

void build_grid3(const mdg_problem_desc &d, Grid3Host &h);

struct Sweep3 {
  Grid3 g{};
  char *d_tab = nullptr;           // all grid tables in one allocation
  double *d_flux = nullptr;        // F0 | F1 | F2, 5 arrays each
  unsigned char *d_bits = nullptr; // own0 | own1 | all0, one byte per zone each
  Tile3 *d_tiles = nullptr;        // zone tiles (the conserved totals)
  int *d_seg = nullptr;            // direction-2 segments, then the first segment of every CTA
  int nseg = 0;
  int *d_row0 = nullptr;           // Grid3::row0
  int *d_runs = nullptr;           // runs | runs | first run of every CTA | the same of direction 1
  size_t runs_cap = 0;             // ints d_runs holds
  size_t run_off[4] = {0, 0, 0, 0};
  int nrun[2] = {0, 0}, nlane[2] = {0, 0};
  int run_len = RUN0;              // longest run asked for
  int run_exact = 0;               // a length fixed by hand, whatever the grid's size (0: fitting_run)
  int run_used = 0;                // the length the lists are cut to
  bool small_rule[3] = {false, false, false};   // face kernel k's launch is a small one (small_by_size)
  int small = -1;                  // the small launches' kernels: by that rule (-1), never, always
  int num_sms = 0;
  // the row structure the run lists are cut from (a copy of the host grid's)
  int n1 = 0, n2 = 0, n3 = 0;
  std::vector<int> nj, rowbase, nk;
  double *d_gmono = nullptr;       // monopole gravity per radial row
  int nt[4] = {0, 0, 0, 0};        // CTAs of face0, face1, face2 and the zone kernels
  int ntot = 0;                    // zone tiles of the conserved totals
  int64_t ncell = 0;
  int64_t bytes = 0;               // device memory held: every allocation goes through take()
  template <typename T> cudaError_t take(T **p, size_t n)
  {
    const cudaError_t e = cudaMalloc(p, n);
    if (e == cudaSuccess) bytes += (int64_t)n;
    return e;
  }
};

static void tiles_of_rows(std::vector<Tile3> &out, int i, int j, int count, int chunk = NT3)
{
  for (int k0 = 0; k0 < count; k0 += chunk) out.push_back(Tile3{i, j, k0, (count - k0 < chunk) ? count - k0 : chunk});
}

// A run list: the runs, the run of each CTA's first lane, and the number of lanes.
struct RunList {
  std::vector<Run3> runs;
  std::vector<int> first;
  int nlane = 0;
};

// The faces of the radial (dir 0) or theta (dir 1) run kernel as runs of at most run_len
// faces; cnt[r] is the number of columns of run r, k0[r] the first.
static void cut_runs(const Sweep3 &w, int dir, int run_len, std::vector<Run3> &runs, std::vector<int> &cnt)
{
  auto njr = [&](int i) { return w.nj[i + NG]; };
  auto row = [&](int i, int j) { return w.rowbase[i + NG] + j + NG; };
  auto dj = [&](int i) { return w.n2 / w.nj[i + NG]; };
  auto dk = [&](int i, int j) { return w.n3 / w.nk[row(i, j)]; };
  if (dir == 0) {
    // faces i in [0, n1] grouped by constant theta resolution, then per theta row j by
    // constant phi resolution, cut into run_len faces
    for (int i = 0; i <= w.n1;) {
      int ie = i + 1;
      while (ie <= w.n1 && dj(ie) == dj(i)) ie++;
      for (int j = 0; j < njr(i); j++) {
        for (int a = i; a < ie;) {
          int b = a + 1;
          while (b < ie && dk(b, j) == dk(a, j)) b++;
          for (int c = a; c < b; c += run_len) {
            runs.push_back(Run3{c, std::min(run_len, b - c), j, 0});
            cnt.push_back(w.nk[row(a, j)]);
          }
          a = b;
        }
      }
      i = ie;
    }
  } else {
    // faces j in [0, nj(i)] of radial row i grouped by constant phi resolution of the face,
    // min(dk(i, j), dk(i, j-1)), cut into run_len faces
    for (int i = 0; i < w.n1; i++) {
      const int nj = njr(i);
      auto mn = [&](int j) { return std::min(dk(i, j), dk(i, j - 1)); };
      for (int a = 0; a <= nj;) {
        int b = a + 1;
        while (b <= nj && mn(b) == mn(a)) b++;
        for (int c = a; c < b; c += run_len) {
          runs.push_back(Run3{c, std::min(run_len, b - c), i, 0});
          cnt.push_back(w.n3 / mn(a));
        }
        a = b;
      }
    }
  }
}

// Longest run, up to run_len faces, for which the grid's lanes still fill the chip (5 CTAs of
// 128 lanes on every SM).  What a lane does once, three pencil entries and a reconstruction,
// is about two faces' worth, so long runs pay where there are lanes enough: ms per step on a
// B200 for runs of 1 / 4 / 8 / 16, 2-D 400 x 256 mixed 0.165 / 0.233 / 0.327 / 0.532 (taken: 1),
// 3-D 100 x 32 x 64 plain FP64 0.416 / 0.456 / 0.578 / 0.867 (1), 128 x 64 x 128 plain FP64 1.547 /
// 1.342 / 1.245 / 1.538 (8), 384 x 128 x 256 plain FP64 9.13 / 7.24 / 6.85 / 6.70 and mixed 7.47 / 5.74 /
// 5.41 / 5.25 (16).
static int fitting_run(const Sweep3 &w, int run_len)
{
  const int64_t fill = (int64_t)(w.num_sms > 0 ? w.num_sms : 148) * 5 * NT3;
  while (run_len > 1 && w.ncell / run_len < fill) run_len = (run_len + 1) / 2;
  return run_len;
}

static void build_runs(const Sweep3 &w, int dir, int run_len, RunList &out)
{
  std::vector<Run3> runs;
  std::vector<int> cnt;
  runs.reserve(w.nk.size() / run_len);
  cnt.reserve(w.nk.size() / run_len);
  cut_runs(w, dir, run_len, runs, cnt);
  out.runs.reserve(runs.size());
  // long runs first (the tail of the launch is made of short ones), neighbouring rows in
  // neighbouring lanes: direction 0 by first face then theta row, direction 1 likewise
  // (a counting sort on length and first face: the runs of a pair already come in row order)
  int rmax = 0;
  for (const Run3 &r : runs) rmax = std::max(rmax, r.r0);
  auto bucket = [&](const Run3 &r) { return (size_t)(run_len - r.nr) * (rmax + 1) + r.r0; };
  std::vector<int> pos((size_t)run_len * (rmax + 1) + 1, 0), ord(runs.size());
  for (const Run3 &r : runs) pos[bucket(r) + 1]++;
  for (size_t q = 1; q < pos.size(); q++) pos[q] += pos[q - 1];
  for (size_t q = 0; q < runs.size(); q++) ord[pos[bucket(runs[q])]++] = (int)q;
  for (int q : ord) {
    Run3 r = runs[q];
    r.l0 = out.nlane;
    out.nlane += cnt[q];
    while ((int)out.first.size() * NT3 < out.nlane) out.first.push_back((int)out.runs.size());
    out.runs.push_back(r);
  }
}

// Direction-2 segments and the first segment of every CTA.
static void build_segs(const Sweep3 &w, std::vector<Seg2> &segs, std::vector<int> &first)
{
  int used = 0, n = 0;   // lanes and segments of the CTA being filled
  for (int i = 0; i < w.n1; i++) {
    for (int j = 0; j < w.nj[i + NG]; j++) {
      const int nf = w.nk[w.rowbase[i + NG] + j + NG] + 1;
      for (int k0 = 0; k0 < nf;) {
        int cnt = std::min(nf - k0, T2);
        if (n == SEG2_MAX) used = n = 0;
        if (used + cnt + 2 > NT3) {
          // does not fit: cut it (two more lanes) where at least 8 faces do, else a new CTA
          const int room = NT3 - used - 2;
          if (room >= 8) cnt = room;
          else used = n = 0;
        }
        if (n == 0) first.push_back((int)segs.size());
        segs.push_back(Seg2{i, j, k0, cnt, used, n});
        used += cnt + 2;
        n++;
        k0 += cnt;
      }
    }
  }
}

// Both run lists for runs of at most run_len faces (exact != 0: of that many, else shorter ones
// where the grid is small), into one device allocation.
static cudaError_t upload_runs(Sweep3 *w, int run_len, int exact)
{
  const int used = exact ? exact : fitting_run(*w, run_len);
  if (used == w->run_used) {
    w->run_len = run_len;
    w->run_exact = exact;
    return cudaSuccess;
  }
  RunList l[2];
  std::vector<int> all;
  size_t off[4];
  for (int d = 0; d < 2; d++) {
    build_runs(*w, d, used, l[d]);
    off[d] = all.size();
    const int *r = reinterpret_cast<const int *>(l[d].runs.data());
    all.insert(all.end(), r, r + sizeof(Run3) / sizeof(int) * l[d].runs.size());
  }
  for (int d = 0; d < 2; d++) {
    off[2 + d] = all.size();
    all.insert(all.end(), l[d].first.begin(), l[d].first.end());
  }
  cudaError_t e = cudaSuccess;
  if (all.size() > w->runs_cap) {
    int *d = nullptr;
    e = w->take(&d, sizeof(int) * all.size());
    if (e != cudaSuccess) return e;
    cudaFree(w->d_runs);
    w->bytes -= (int64_t)(sizeof(int) * w->runs_cap);
    w->d_runs = d;
    w->runs_cap = all.size();
  }
  e = cudaMemcpy(w->d_runs, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = setup_landed();
  if (e != cudaSuccess) return e;
  for (int q = 0; q < 4; q++) w->run_off[q] = off[q];
  for (int d = 0; d < 2; d++) {
    w->nt[d] = (int)l[d].first.size();
    w->nrun[d] = (int)l[d].runs.size();
    w->nlane[d] = l[d].nlane;
  }
  w->run_len = run_len;
  w->run_exact = exact;
  w->run_used = used;
  return cudaSuccess;
}

int sweep3_set_run_length(Sweep3 *w, int run_length, int exact, std::string &why)
{
  if (run_length < 1 || run_length > 64) { why = "run_length out of [1, 64]"; return MDG_ERR_INVALID; }
  if (exact < 0 || exact > 64) { why = "exact run length out of [0, 64]"; return MDG_ERR_INVALID; }
  const cudaError_t e = upload_runs(w, run_length, exact);
  if (e != cudaSuccess) {
    why = cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? MDG_ERR_OUTOFMEM : MDG_ERR_CUDA;
  }
  return MDG_OK;
}
void sweep3_set_small(Sweep3 *w, int small) { w->small = small; }
static bool small_launch(const Sweep3 &w, int k)
{
  return w.small >= 0 ? w.small == 1 : w.small_rule[k];
}
// Which launches are small is settled once, with the run length that the grid's size gives: the two
// variants of a mixed kernel contract differently, and the results are not to depend on the run
// length that is set later.
static void small_by_size(Sweep3 *w)
{
  for (int k = 0; k < 3; k++) w->small_rule[k] = w->nt[k] <= F3MINB_SMALL * w->num_sms;
}
void sweep3_run_shape(const Sweep3 *w, int *exact, int *used, int *small)
{
  *exact = w->run_exact;
  *used = w->run_used;
  *small = 0;
  for (int k = 0; k < 3; k++) *small |= small_launch(*w, k) ? 1 << k : 0;
}

int sweep3_create(const mdg_problem_desc &d, Sweep3 **out, std::string &why)
{
  *out = nullptr;
  Grid3Host h;
  build_grid3(d, h);
  if (h.nlev1 > G3_MAXLEV || h.nlev2 > G3_MAXLEV) { why = "too many refinement levels"; return MDG_ERR_INVALID; }
  Sweep3 *w = new Sweep3();
  w->ncell = h.ncell;
  // push() flux addresses of every interior row (the fan-in rules of push3_kernel), in zone
  // order, with the first zone of each row and the row of each CTA's first zone
  std::vector<PushRow3> prow;
  std::vector<int64_t> rowcell;
  std::vector<int> row0;
  prow.reserve((size_t)h.nij);
  rowcell.reserve((size_t)h.nij);
  for (int i = 0; i < h.n1; i++) {
    for (int j = 0; j < h.njr(i); j++) {
      PushRow3 r{};
      const int ij = h.row(i, j);
      const int dji = h.dj(i), djo = h.dj(i + 1), dkij = h.dk(i, j);
      const int jp = j * dji / djo;
      r.nf0o = (djo < dji) ? dji / djo : 1;
      for (int q = 0; q < r.nf0o; q++) {
        r.nkp[q] = dkij / h.dk(i + 1, jp + q);
        r.f0o[q] = h.f0[h.row(i + 1, jp + q)];
      }
      r.f0i = h.f0[ij];
      const int dkp = h.dk(i, j + 1), dkm = h.dk(i, j - 1);
      r.f1o = h.f1[h.row(i, j + 1)];
      r.f1i = h.f1[ij];
      r.mo = (dkp > dkij) ? 1 : (dkp < dkij ? 2 : 0);
      r.mi = (dkm < dkij) ? 1 : 0;
      r.f2 = h.ndim == 3 ? h.f2[ij] : 0;
      r.i = i;
      r.j = j;
      r.ij = ij;
      while ((int64_t)row0.size() * NT3 < h.cell[ij] + h.nk[ij]) row0.push_back((int)prow.size());
      prow.push_back(r);
      rowcell.push_back(h.cell[ij]);
    }
  }
  // one allocation for every table, each part 256-byte aligned
  std::vector<std::pair<const void *, size_t>> parts = {
      {h.nj.data(), h.nj.size() * sizeof(int)},         {h.rowbase.data(), h.rowbase.size() * sizeof(int)},
      {h.nk.data(), h.nk.size() * sizeof(int)},         {h.cell.data(), h.cell.size() * sizeof(int64_t)},
      {h.f0.data(), h.f0.size() * sizeof(int64_t)},     {h.f1.data(), h.f1.size() * sizeof(int64_t)},
      {h.f2.data(), h.f2.size() * sizeof(int64_t)},     {h.geo.data(), h.geo.size() * sizeof(double)},
      {h.rc0.data(), h.rc0.size() * sizeof(double)},    {h.rc1.data(), h.rc1.size() * sizeof(double)},
      {h.rc2.data(), h.rc2.size() * sizeof(double)},    {h.xc1.data(), h.xc1.size() * sizeof(double)},
      {h.xc2.data(), h.xc2.size() * sizeof(double)},    {h.sth.data(), h.sth.size() * sizeof(double)},
      {h.cth.data(), h.cth.size() * sizeof(double)},    {h.sphc.data(), h.sphc.size() * sizeof(double)},
      {h.cphc.data(), h.cphc.size() * sizeof(double)},  {h.sphl.data(), h.sphl.size() * sizeof(double)},
      {h.cphl.data(), h.cphl.size() * sizeof(double)},  {h.mx0.data(), h.mx0.size() * sizeof(float)},
      {h.mx1.data(), h.mx1.size() * sizeof(float)},     {h.mx2.data(), h.mx2.size() * sizeof(float)},
      {h.medge.data(), h.medge.size() * sizeof(double)},    {prow.data(), prow.size() * sizeof(PushRow3)},
      {rowcell.data(), rowcell.size() * sizeof(int64_t)}};
  std::vector<size_t> off(parts.size());
  size_t tot = 0;
  for (size_t q = 0; q < parts.size(); q++) {
    off[q] = tot;
    tot += (parts[q].second + 255) / 256 * 256;
  }
  auto fail3 = [&](cudaError_t e) {
    why = cudaGetErrorString(e);
    cudaFree(w->d_tab); cudaFree(w->d_flux); cudaFree(w->d_bits); cudaFree(w->d_tiles); cudaFree(w->d_gmono);
    cudaFree(w->d_runs); cudaFree(w->d_seg); cudaFree(w->d_row0);
    delete w;
    return e == cudaErrorMemoryAllocation ? MDG_ERR_OUTOFMEM : MDG_ERR_CUDA;
  };
  cudaError_t e = w->take(&w->d_tab, tot);
  if (e != cudaSuccess) return fail3(e);
  // part by part: packing them on the host first took a fifth of a (r, theta) grid's set-up
  for (size_t q = 0; q < parts.size() && e == cudaSuccess; q++)
    if (parts[q].second) e = cudaMemcpy(w->d_tab + off[q], parts[q].first, parts[q].second, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return fail3(e);
  Grid3 &g = w->g;
  g.ndim = h.ndim;
  g.n1 = h.n1; g.n2 = h.n2; g.n3 = h.n3;
  g.bc_lo0 = d.bc_lo[0]; g.bc_hi0 = d.bc_hi[0]; g.bc_lo1 = d.bc_lo[1]; g.bc_hi1 = d.bc_hi[1];
  g.bc_lo2 = d.bc_lo[2]; g.bc_hi2 = d.bc_hi[2];
  g.dx0 = d.dx[0]; g.dx1 = d.dx[1]; g.dx2 = d.dx[2];
  g.nij = h.nij; g.ncell = h.ncell; g.nf0 = h.nf0; g.nf1 = h.nf1; g.nf2 = h.nf2;
  g.cols1 = h.cols1; g.cols2 = h.cols2;
  for (int l = 0; l < G3_MAXLEV; l++) { g.rc1_base[l] = h.rc1_base[l]; g.rc2_base[l] = h.rc2_base[l]; }
  char *b = w->d_tab;
  g.nj = (const int *)(b + off[0]); g.rowbase = (const int *)(b + off[1]); g.nk = (const int *)(b + off[2]);
  g.cell = (const int64_t *)(b + off[3]); g.f0 = (const int64_t *)(b + off[4]);
  g.f1 = (const int64_t *)(b + off[5]); g.f2 = (const int64_t *)(b + off[6]);
  g.geo = (const double *)(b + off[7]); g.rc0 = (const double *)(b + off[8]);
  g.rc1 = (const double *)(b + off[9]); g.rc2 = (const double *)(b + off[10]);
  g.xc1 = (const double *)(b + off[11]); g.xc2 = (const double *)(b + off[12]);
  g.sth = (const double *)(b + off[13]); g.cth = (const double *)(b + off[14]);
  g.sphc = (const double *)(b + off[15]); g.cphc = (const double *)(b + off[16]);
  g.sphl = (const double *)(b + off[17]); g.cphl = (const double *)(b + off[18]);
  g.mx0 = (const float *)(b + off[19]); g.mx1 = (const float *)(b + off[20]); g.mx2 = (const float *)(b + off[21]);
  g.medge = (const double *)(b + off[22]);
  g.prow = (const PushRow3 *)(b + off[23]);
  g.rowcell = (const int64_t *)(b + off[24]);
  g.nrow = (int)prow.size();
  g.x0 = d.startx[0];
  g.mono = d.monopole;
  e = w->take(&w->d_gmono, sizeof(double) * (size_t)h.n1);
  if (e != cudaSuccess) return fail3(e);
  g.gmono = w->d_gmono;
  // flux arrays, shock bits
  e = w->take(&w->d_flux, sizeof(double) * NPRIM * (size_t)(h.nf0 + h.nf1 + h.nf2));
  if (e != cudaSuccess) return fail3(e);
  e = w->take(&w->d_bits, (size_t)3 * h.ncell);
  if (e != cudaSuccess) return fail3(e);
  e = cudaMemset(w->d_bits, 0, (size_t)3 * h.ncell);
  if (e != cudaSuccess) return fail3(e);
  // tiles of each kernel
  std::vector<Tile3> tc;
  w->n1 = h.n1; w->n2 = h.n2; w->n3 = h.n3;
  w->nj = h.nj; w->rowbase = h.rowbase; w->nk = h.nk;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&w->num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    w->num_sms = 0;
  for (int i = 0; i < h.n1; i++)
    for (int j = 0; j < h.njr(i); j++) tiles_of_rows(tc, i, j, h.nk[h.row(i, j)]);
  w->ntot = (int)tc.size();
  w->nt[3] = (int)row0.size();
  e = w->take(&w->d_row0, sizeof(int) * row0.size());
  if (e != cudaSuccess) return fail3(e);
  e = cudaMemcpy(w->d_row0, row0.data(), sizeof(int) * row0.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return fail3(e);
  g.row0 = w->d_row0;
  e = w->take(&w->d_tiles, sizeof(Tile3) * tc.size());
  if (e != cudaSuccess) return fail3(e);
  e = cudaMemcpy(w->d_tiles, tc.data(), sizeof(Tile3) * tc.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return fail3(e);
  if (h.ndim == 3) {
    std::vector<Seg2> segs;
    std::vector<int> first, all;
    build_segs(*w, segs, first);
    w->nt[2] = (int)first.size();
    w->nseg = (int)segs.size();
    const int *q = reinterpret_cast<const int *>(segs.data());
    all.assign(q, q + sizeof(Seg2) / sizeof(int) * segs.size());
    all.insert(all.end(), first.begin(), first.end());
    e = w->take(&w->d_seg, sizeof(int) * all.size());
    if (e != cudaSuccess) return fail3(e);
    e = cudaMemcpy(w->d_seg, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail3(e);
  }
  e = upload_runs(w, RUN0, 0);
  if (e != cudaSuccess) return fail3(e);
  small_by_size(w);
  *out = w;
  return MDG_OK;
}

void sweep3_destroy(Sweep3 *w)
{
  if (!w) return;
  cudaFree(w->d_tab); cudaFree(w->d_flux); cudaFree(w->d_bits); cudaFree(w->d_tiles); cudaFree(w->d_gmono);
  cudaFree(w->d_runs); cudaFree(w->d_seg); cudaFree(w->d_row0);
  delete w;
}

int64_t sweep3_ncell(const Sweep3 *w) { return w->ncell; }
int64_t sweep3_bytes(const Sweep3 *w) { return w->bytes; }

// Kernel launches of one RK stage of the single 3-D problem (slot 0).
void launch_stage3d(int stage, bool mixed, Sweep3 *w, const ProbDev *probs, ProbTime *times, StateSoA sst,
                    StateSoA sn, StateSoA out, cudaStream_t st)
{
  const Grid3 &g = w->g;
  double *F0 = w->d_flux, *F1 = F0 + NPRIM * g.nf0, *F2 = F1 + NPRIM * g.nf1;
  unsigned char *own = w->d_bits + (size_t)stage * g.ncell, *all0 = w->d_bits + (size_t)2 * g.ncell;
  const Run3 *r0 = reinterpret_cast<const Run3 *>(w->d_runs + w->run_off[0]);
  const Run3 *r1 = reinterpret_cast<const Run3 *>(w->d_runs + w->run_off[1]);
  const int *l0 = w->d_runs + w->run_off[2], *l1 = w->d_runs + w->run_off[3];
  const Seg2 *segs = reinterpret_cast<const Seg2 *>(w->d_seg);
  const int *l2 = w->d_seg + sizeof(Seg2) / sizeof(int) * w->nseg;
  if (stage == 0) cudaMemsetAsync(all0, 0, (size_t)g.ncell, st);
  if (g.mono) {
    shell_mass3_kernel<<<(g.n1 + 127) / 128, 128, 0, st>>>(times, g, sst);
    monopole_profile3_kernel<<<1, 32, 0, st>>>(times, g);
  }
  const FaceLaunch3 f{{w->nt[0], w->nt[1], w->nt[2]}, {small_launch(*w, 0), small_launch(*w, 1), small_launch(*w, 2)}, {r0, r1}, {l0, l1, l2}, {w->nrun[0], w->nrun[1]},
                      {w->nlane[0], w->nlane[1]}, w->nseg, segs, {F0, F1, F2}, own, all0};
  if (mixed) launch_faces3_mixed(stage, f, probs, times, g, sst, st);
  else if (stage == 0) launch_faces3<0, false>(f, probs, times, g, sst, st);
  else launch_faces3<1, false>(f, probs, times, g, sst, st);
  if (stage == 0) push3_kernel<0><<<w->nt[3], NT3, 0, st>>>(probs, times, g, sst, sn, out, F0, F1, F2);
  else push3_kernel<1><<<w->nt[3], NT3, 0, st>>>(probs, times, g, sst, sn, out, F0, F1, F2);
}

void launch_totals3(Sweep3 *w, StateSoA s, double *out, cudaStream_t st)
{
  totals3_kernel<<<1, 256, 0, st>>>(w->g, w->d_tiles, w->ntot, s, out);
}

void launch_initial_estimate3(Sweep3 *w, const ProbDev *probs, ProbTime *times, StateSoA s, cudaStream_t st)
{
  estimate3_kernel<<<w->nt[3], NT3, 0, st>>>(probs, times, w->g, s);
}

}  // namespace mdg
