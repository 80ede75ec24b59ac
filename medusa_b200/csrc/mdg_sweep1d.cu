// Fused 1-D RK stage kernel (plain FP64).
//
// One CTA advances one tile of TILE1 = 126 zones of one problem through a whole RK
// stage: it stages the 130-zone pencil (tile + 2 ghost zones each side) in shared
// memory, reconstructs every zone ONCE (the reference reconstructs each zone twice,
// once per adjacent face: step.c:501-547), solves the 127 face Riemann problems, and
// applies push() (step.c:380-470) to its 126 zones.  Boundary zones are never stored:
// they are produced on load by the boundary kinds of reset_boundaries_gpu (bc.c:705-1422)
// as index maps.  The CFL minimum (face terms step.c:560, source terms step.c:393, and in
// the second stage the zone terms of the next estimate_dt, step.c:177-187) is reduced
// per CTA by warp reductions and folded into the problem's accumulator with one atomic.
//
// Many problems of different sizes are advanced by one launch: the grid is a list of
// (problem, tile) work items.
//
// Small problems (at most 16 tiles, 2016 zones) can instead be advanced by the resident
// stepper: one thread-block cluster per problem, one CTA per tile, runs the whole step
// sequence of many steps in one launch -- the dt rules, both RK stages and the time
// update, separated by cluster barriers -- where the per-phase path pays three dependent
// launches per step.  It runs the same tile code, so the two paths agree bit for bit.
#include "mdg_hydro.cuh"
#include "mdg_kernels.cuh"
#include "mdg_load1d.cuh"
#include "mdg_tma.cuh"
#include "mdg_timeloop.cuh"
#include <cooperative_groups.h>

namespace mdg {

// TMA: the tile's reconstruction coefficients (all RC_TMA_ROWS rows) and face/zone geometry
// (GF_TMA_ROWS rows) arrive in shared memory by two tensor loads issued at the start,
// which overlap the state loads; otherwise every field is read from the tables in HBM
// when used.  The results are the same.
// One RK stage of one tile, run by the NT1 x G threads of a CTA: thread t of group 0 does zone
// t of the tile; with G = 4 the groups share the six variables' reconstructions of every zone
// (density / internal energy / v1 and v2 / pressure and v3).  dt, t_bc: the step and the time the
// boundaries see; minacc: the CFL accumulator (OWN: this CTA's alone); T: the problem's record (error mark).  tm: the
// tensor maps of the tables (a __grid_constant__ kernel parameter; not read without TMA).
template <int STAGE, bool TMA, int G, bool OWN>
__device__ __forceinline__ void stage1d_tile(const ProbDev &P, ProbTime *T, double dt, double t_bc,
                                             unsigned long long *minacc, const Tile tile, const Tables &tb,
                                             const StateSoA &sst, const StateSoA &sn, const StateSoA &out,
                                             const TmaTables1d &tm)
{
  static_assert(G == 1 || (G == 4 && !TMA), "one thread per zone, or four without TMA");
  __shared__ double sv[6][NT1 + 2];     // stage-state pencil: 5 primitives + pressure
  __shared__ double sred[32];
  __shared__ __align__(128) double s_rc[TMA ? RC_TMA_ROWS : 1][TMA ? TMA_COLS1 : 1];
  __shared__ __align__(128) double s_geo[TMA ? GF_TMA_ROWS : 1][TMA ? TMA_COLS1 : 1];
  __shared__ __align__(8) uint64_t s_bar;
  // right face values of each reconstructed zone and the face fluxes; with TMA they
  // reuse the reconstruction rows, which are dead once every zone is reconstructed
  __shared__ double sar_own[TMA ? 1 : 6][NT1];
  __shared__ double sfl_own[TMA ? 1 : NPRIM][NT1];
  static_assert(!TMA || (6 + NPRIM) * NT1 <= RC_TMA_ROWS * TMA_COLS1, "exchange buffers fit the recon rows");
  double (*sar)[NT1] = TMA ? reinterpret_cast<double(*)[NT1]>(&s_rc[0][0]) : sar_own;
  double (*sfl)[NT1] = TMA ? reinterpret_cast<double(*)[NT1]>(&s_rc[0][0] + 6 * NT1) : sfl_own;

  __shared__ double sal[G > 1 ? 6 : 1][G > 1 ? NT1 : 1];   // left face values (G > 1: other groups' threads)
  const int t = G > 1 ? threadIdx.x % NT1 : threadIdx.x, grp = G > 1 ? threadIdx.x / NT1 : 0;
  const int n1 = P.n1;
  const int z = tile.i0 - 1 + t;           // zone reconstructed by this thread
  const double *rc = tb.rc0;
  const int64_t rcs = tb.rc0_stride;
  const double *geo = tb.geo;
  const int64_t gs = tb.geo_stride;
  // first table column of the box: the column of zone i0-1 rounded down to even (TMA
  // start coordinates are 16-byte aligned); a table column c sits at box column c - bx
  const int64_t bx = (P.geo_off + NG + tile.i0 - 1) & ~int64_t(1);
  if (TMA) {
    if (t == 0) mbar_init(&s_bar, 1);
    __syncthreads();
    if (t == 0) {
      mbar_arrive_expect_tx(&s_bar, (unsigned)((RC_TMA_ROWS + GF_TMA_ROWS) * TMA_COLS1 * sizeof(double)));
      tma_load_2d(&s_rc[0][0], &tm.rc, (int)bx, 0, &s_bar);
      tma_load_2d(&s_geo[0][0], &tm.geo, (int)bx, 0, &s_bar);
    }
  }
  // geometry field f of table column c (faces and zones of this tile)
  auto gf = [&](int f, int64_t c) -> double {
    if (TMA) return s_geo[f][c - bx];
    return __ldg(geo + f * gs + c);
  };

  if (grp == 0) {
    double w[6];
    load_cell_1d(P, sst, rc, rcs, z, t_bc, w);
#pragma unroll
    for (int v = 0; v < 6; v++) sv[v][t + 1] = w[v];
  }
  // the outer columns (with several groups, by threads that load nothing else)
  if (t == 0 && grp == G - 1) {
    double w2[6];
    load_cell_1d(P, sst, rc, rcs, tile.i0 - 2, t_bc, w2);
#pragma unroll
    for (int v = 0; v < 6; v++) sv[v][0] = w2[v];
  }
  if (t == NT1 - 1 && grp == G - 1) {
    double w2[6];
    load_cell_1d(P, sst, rc, rcs, tile.i0 + NT1 - 1, t_bc, w2);
#pragma unroll
    for (int v = 0; v < 6; v++) sv[v][NT1 + 1] = w2[v];
  }
  if (TMA) {
    // the tables have landed (bounded wait: a copy that never completes flags the
    // problem and the CTA leaves after waiting once more, as bounded)
    const bool ok = mbar_wait(&s_bar, 0);
    if (__syncthreads_or(!ok)) {
      if (t == 0) T->err = MDG_ERR_INTERNAL;
      mbar_wait(&s_bar, 0);
      return;
    }
  }
  __syncthreads();

  // reconstruct zone z once (interp(), reconstruct.c:225-279); Gamma is the constant
  // adiabatic index, which every order reconstructs to itself.
  double al[7], ar[7];
  if (G > 1) {
    const int zc = z < -1 ? -1 : (z > n1 ? n1 : z);
    const RcView<double, true> g{rc + P.geo_off + zc + NG, rcs};
    const int first = grp == 3 ? 5 : grp, second = grp < 2 ? -1 : grp + 1;
#pragma unroll 1
    for (int v = first; v >= 0; v = (v == first) ? second : -1) {
      const FacePair o = recon_var(P.interp_order, sv[v][t], sv[v][t + 1], sv[v][t + 2], g);
      sal[v][t] = o.al;
      sar[v][t] = o.ar;
    }
  } else {
    int zc = z < -1 ? -1 : (z > n1 ? n1 : z);
    const int64_t c = P.geo_off + zc + NG;
    const RcView<double, !TMA> g{TMA ? &s_rc[0][c - bx] : rc + c, TMA ? (int64_t)TMA_COLS1 : rcs};
    recon_vars<6>(P.interp_order, g, [&](int v, int q) { return sv[v][t + q]; },
                  [&](int v, double lo, double hi) { al[v] = lo; ar[v] = hi; });
    al[6] = P.gam; ar[6] = P.gam;
  }
  if (TMA) __syncthreads();   // every zone reconstructed: the recon rows may be overwritten
  if (G == 1) {
#pragma unroll
    for (int v = 0; v < 6; v++) sar[v][t] = ar[v];
  }
  __syncthreads();
  if (G > 1 && grp == 0) {
#pragma unroll
    for (int v = 0; v < 6; v++) al[v] = sal[v][t];
    al[6] = P.gam;
  }

  double lmin = 1.0e300;
  double smax = 0.0, nmin = 1.0e300, lmax = 0.0;
  const GamConst<double> gc = gam_const(P.gam);
  // face z: between zones z-1 and z (pl = right state of z-1, pr = left state of z)
  const bool face_ok = (t >= 1) && (z >= 0) && (z <= n1);
  if (t >= 1 && grp == 0) {
    double pl[7], flux[NPRIM], sig;
#pragma unroll
    for (int v = 0; v < 6; v++) pl[v] = sar[v][t - 1];
    pl[6] = P.gam;
    FaceGeom<double> fg;
    int zf = z < 0 ? 0 : (z > n1 ? n1 : z);
    const int64_t gi = P.geo_off + zf + NG;
    fg.area = gf(GF_AREA, gi);
    fg.scale = gf(GF_FSCALE, gi);
    fg.g0 = gf(GF_FG0, gi);
    fg.g1 = gf(GF_FG1, gi);
    fg.g2 = gf(GF_FG2, gi);
    riemann_hllc<0, false, double>(pl, al, fg, gc, flux, sig);
#pragma unroll
    for (int v = 0; v < NPRIM; v++) sfl[v][t] = flux[v];
    if (face_ok) smax = tmax(smax, fabs(sig));
  }
  __syncthreads();

  // push() for zone z (step.c:380-470)
  if (grp == 0 && t >= 1 && t <= NT1 - 2 && z >= 0 && z < n1) {
    const int64_t gi = P.geo_off + z + NG;
    const int64_t cell = P.cell_off + z;
    double ph[NPRIM], pn[NPRIM], u[NPRIM], uh[NPRIM], src[NPRIM], divF[NPRIM], pf[NPRIM];
#pragma unroll
    for (int v = 0; v < NPRIM; v++) ph[v] = sv[v][t + 1];
    if (STAGE == 0) {
#pragma unroll
      for (int v = 0; v < NPRIM; v++) pn[v] = ph[v];
    } else {
#pragma unroll
      for (int v = 0; v < NPRIM; v++) pn[v] = sn.v[v][cell];
    }
    const double gc0 = gf(GF_G0, gi), gc1 = gf(GF_G1, gi), gc2 = gf(GF_G2, gi);
    // geometric source terms from the stage state (rad_fluid.c:164-192, fluid.c:56-73)
    if (P.has_src) {
      geo_sources_1d(geo, gs, gi, P.sparse_conn != 0, ph, sv[5][t + 1], gc0, gc1, gc2, src);
    } else {
#pragma unroll
      for (int v = 0; v < NPRIM; v++) src[v] = 0.0;
    }
    if (P.grav_on) add_fixed_gravity(ph, P.grav, gc0, gc1, gc2, 1, src);
    if (P.mono) {
      // mass flux density at the outer and inner face (gravity.c:380-401)
      double vr = 0.0, area = 0.0;
      vr += sfl[RHO][t + 1];
      area += gf(GF_AREA, gi + 1) + 1.0e-16;
      vr /= area;
      const double vl = sfl[RHO][t] / (gf(GF_AREA, gi) + 1.0e-16);
      add_monopole_gravity(ph[RHO], tb.gmono[P.mono_off + z], vl, vr, P.x0 + z * P.dx0, P.dx0,
                           __ldg(rc + RC_B0 * rcs + gi), __ldg(rc + RC_G0 * rcs + gi), src);
    }
    p_to_u(pn, u, gc0, gc1, gc2);
    p_to_u(ph, uh, gc0, gc1, gc2);
    if (P.has_src || P.grav_on || P.mono) lmin = tmin(lmin, dt_source_control(pn, u, src));
    else nmin = tmin(nmin, src_dt_numerator_min(pn, u));   // zero sources: shared denominator
#pragma unroll
    for (int v = 0; v < NPRIM; v++) { divF[v] = 0.0; divF[v] += sfl[v][t + 1]; divF[v] -= sfl[v][t]; }
    const double vol = gf(GF_VOL, gi);
    const double pfact = STAGE ? 0.5 : 1.0, phfact = STAGE ? 0.5 : 0.0, ffact = STAGE ? 0.5 : 1.0;
    double dv[NPRIM];
    quotients<NPRIM>(divF, vol, dv);
#pragma unroll
    for (int v = 0; v < NPRIM; v++) {
      double ddt = dv[v] - src[v];
      u[v] = pfact * u[v] + phfact * uh[v] - ffact * dt * ddt;
    }
    u_to_p(u, pf, gf(GF_GC0, gi), gf(GF_GC1, gi), gf(GF_GC2, gi), P.floors != 0, P.rho_floor, P.e_floor);
#pragma unroll
    for (int v = 0; v < NPRIM; v++) out.v[v][cell] = pf[v];
    flag_nonfinite(pf, T);
    if (STAGE == 1) {
      // zone term of the next estimate_dt (step.c:177-187): velocity of the new state,
      // sound speed of the stage state (sim_eos was last filled from sim_ph)
      const double cs = sqrt(P.gam * sv[5][t + 1] / ph[RHO]);
      double local_dt = 0.0;
      local_dt += (fabs(pf[U1]) + cs / gf(GF_S00, gi)) / P.dx0;
      lmax = tmax(lmax, local_dt);
    }
  }
  // min of dx/|sig| over faces, of the zero-source limits and of 1/local_dt, each taken
  // on its numerator or denominator (monotone division, see src_dt_numerator_min)
  if (grp == 0) {
    lmin = tmin(lmin, P.dx0 / smax);
    lmin = tmin(lmin, src_dt_from_numerator(nmin));
    if (STAGE == 1) lmin = tmin(lmin, 1.0 / lmax);
  }
  block_min_to<OWN>(lmin, minacc, sred);
}

template <int STAGE, bool TMA>
__global__ void __launch_bounds__(NT1)
stage1d_kernel(const ProbDev *__restrict__ probs, ProbTime *__restrict__ times,
               const Tile *__restrict__ tiles, Tables tb, StateSoA sst, StateSoA sn, StateSoA out,
               const __grid_constant__ TmaTables1d tm)
{
  const Tile tile = tiles[blockIdx.x];
  ProbTime *T = times + tile.prob;
  if (T->done) return;   // past tmax: the time loop has ended (CTA-uniform)
  stage1d_tile<STAGE, TMA, 1, false>(probs[tile.prob], T, T->dt, STAGE ? T->t_bc1 : T->t, &T->minacc, tile, tb, sst, sn, out,
                              tm);
}

// The resident stepper: nsteps steps of every problem, cluster c advancing problem c with
// CTA r on the tile of zones [126 r, 126 r + 126) (CTAs past the last zone only take part
// in the barriers).  Every CTA keeps the problem's time record in shared memory and runs the
// time rules on its own copy (the same arithmetic on the same numbers, so the copies agree);
// what the CTAs exchange is the state, through global memory, and their tiles' CFL minima, which
// each CTA keeps in its shared memory, in two words that take turns, and reads from the others'
// (distributed shared memory, plain loads).  Each step: the dt rules, stage 0 (p -> ph), a
// cluster barrier, stage 1 (ph, p -> p), a cluster barrier, the time update (the barriers release
// and acquire at cluster scope).  A step's word is read after its last barrier and cleared by
// its owner after the next one, one barrier before its next use.  Every CTA
// takes the same barriers: the loop runs nsteps iterations unless the problem's loop has ended
// (t >= tmax), which every copy of the record says at the same step.  CTA 0 writes the record
// back at the end.
//
// G threads per zone: a stage of so few zones is a chain of dependent FP64 operations, and the
// six reconstructions were a third of it one after the other.  With a CTA per SM (G = 4, all
// clusters resident at once) the groups run them side by side.  Together with the record
// copies (two barriers a step for three, no thread that the others wait for): Sod 1024 23.5 ->
// 21.1 us per step.
//
// PER_SM: CTAs per SM asked of the compiler.  One thread per zone comes with 3 (162 registers) and
// with 4 (128), see resident1d_cluster_size.
template <int G, int PER_SM>
__global__ void __launch_bounds__(NT1 * G, PER_SM)
resident1d_kernel(const ProbDev *__restrict__ probs, ProbTime *__restrict__ times, Tables tb, StateSoA p,
                  StateSoA ph, int nsteps, int *err, const __grid_constant__ TmaTables1d none)
{
  namespace cg = cooperative_groups;
  __shared__ ProbTime rec;
  __shared__ unsigned long long acc[2];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int m = (int)(blockIdx.x / cl.num_blocks());
  const ProbDev &P = probs[m];
  const Tile tile{m, rank * TILE1, 0, 0};
  const bool active = tile.i0 < P.n1, first = threadIdx.x == 0;
  const int lane = (int)threadIdx.x, ncta = (int)cl.num_blocks();
  // the smallest of the CTAs' words w (run by warp 0)
  auto cluster_min = [&](int w) {
    const unsigned long long v = lane < ncta ? *cl.map_shared_rank(acc + w, lane < ncta ? lane : 0) : ~0ull;
    return warp_min_ord(v);
  };
  if (first) {
    rec = times[m];
    acc[0] = acc[1] = dbl_to_ord(1.0e100);
  }
  cl.sync();
  int k = 0;
  for (; k < nsteps; k++) {
    unsigned long long *mine = acc + (k & 1), *last = acc + ((k + 1) & 1);
    if (threadIdx.x < 32) {
      const unsigned long long min_last = k > 0 ? cluster_min((k + 1) & 1) : 0ull;
      if (first) {
        if (k > 0) rec.minacc = min_last;
        dt_finalize_one(P, &rec, err);
      }
    }
    __syncthreads();
    if (rec.done) break;
    if (active) stage1d_tile<0, false, G, true>(P, times + m, rec.dt, rec.t, mine, tile, tb, p, p, ph, none);
    cl.sync();
    if (first) *last = dbl_to_ord(1.0e100);                // every CTA has read it
    if (active) stage1d_tile<1, false, G, true>(P, times + m, rec.dt, rec.t_bc1, mine, tile, tb, ph, p, p, none);
    cl.sync();
    if (first) finish_one(&rec);
  }
  const unsigned long long min_end = threadIdx.x < 32 ? cluster_min((k + 1) & 1) : 0ull;
  if (first && rank == 0) {
    if (k < nsteps) finish_one(&rec);                      // the loop has ended: as a step past it
    else rec.minacc = min_end;
    ProbTime *T = times + m;
    T->t = rec.t; T->dt = rec.dt; T->dtold = rec.dtold; T->t_bc1 = rec.t_bc1; T->t_next = rec.t_next;
    T->minacc = rec.minacc; T->istep = rec.istep; T->dt_ready = rec.dt_ready; T->done = rec.done;
    if (rec.err) T->err = rec.err;                         // (the tiles mark non-finite states in *T)
  }
  cl.sync();                                               // the CTAs' words outlive every reader
}

static void (*resident1d_fn(Resident1d kind))(const ProbDev *, ProbTime *, Tables, StateSoA, StateSoA, int, int *,
                                              const TmaTables1d)
{
  return kind == Resident1d::wide    ? resident1d_kernel<4, 1>
         : kind == Resident1d::dense ? resident1d_kernel<1, 4>
                                     : resident1d_kernel<1, 3>;
}

static cudaLaunchConfig_t resident1d_config(int cs, int nprob, Resident1d kind, cudaStream_t st,
                                            cudaLaunchAttribute *attr)
{
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)(cs * nprob), 1, 1);
  c.blockDim = dim3(kind == Resident1d::wide ? 4 * NT1 : NT1, 1, 1);
  c.dynamicSmemBytes = 0;
  c.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  c.attrs = attr;
  c.numAttrs = 1;
  return c;
}

// Clusters of cs CTAs that the device holds at once (0: none, or the query failed).
static int resident1d_clusters(int cs, Resident1d kind)
{
  const void *f = (const void *)resident1d_fn(kind);
  if (cs > 8 && cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t c = resident1d_config(cs, 1, kind, nullptr, attr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, f, &c) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int resident1d_cluster_size(int max_tiles, int nprob, Resident1d *kind)
{
  *kind = Resident1d::narrow;
  if (max_tiles < 1 || max_tiles > RESIDENT1D_MAX_TILES) return 0;
  int cs = 1;
  while (cs < max_tiles) cs <<= 1;
  const int narrow = resident1d_clusters(cs, Resident1d::narrow), dense = resident1d_clusters(cs, Resident1d::dense);
  if (narrow < 1 && dense < 1) return 0;
  // One thread per zone: the clusters run in waves, so 4 CTAs per SM where that takes fewer waves,
  // else the 3 whose 162 registers are 3-8 % faster.  us per step on a B200, 3 and 4 CTAs per SM: 592
  // problems of up to 126 zones 58 / 38, 48 of up to 1500 (16 CTAs each) 80 / 61, 37 of up to 2000 58 / 64, 100
  // of up to 480 30.0 / 31.1, 12 of up to 250 24.8 / 25.4.
  auto waves = [&](int held) { return held < 1 ? nprob + 1 : (nprob + held - 1) / held; };
  if (waves(dense) < waves(narrow)) *kind = Resident1d::dense;
  // four threads per zone, a whole SM per CTA, for up to 16 CTAs: a ninth of the device, so that
  // several solvers can run beside each other.  (Four solvers of 9 problems of 91-450 zones, 36
  // CTAs each, took 46 us a step that way and 30 us with one thread per zone.)
  if (cs * nprob <= 16 && resident1d_clusters(cs, Resident1d::wide) >= nprob) *kind = Resident1d::wide;
  return cs;
}

cudaError_t launch_resident1d(int cs, Resident1d kind, int nprob, const ProbDev *probs, ProbTime *times,
                              const Tables &tb, StateSoA p, StateSoA ph, int nsteps, int *err, cudaStream_t st)
{
  if (nsteps <= 0 || nprob <= 0) return cudaSuccess;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t c = resident1d_config(cs, nprob, kind, st, attr);
  static const TmaTables1d none{};
  return cudaLaunchKernelEx(&c, resident1d_fn(kind), probs, times, tb, p, ph, nsteps, err, none);
}

void launch_stage1d(int stage, const ProbDev *probs, ProbTime *times, const Tile *tiles, int ntiles,
                    const Tables &tb, StateSoA sst, StateSoA sn, StateSoA out, cudaStream_t st,
                    const TmaTables1d *tm)
{
  if (ntiles <= 0) return;
  static const TmaTables1d none{};
  const bool tma = tm && tm->valid;
  const TmaTables1d &m = tma ? *tm : none;
  if (stage == 0 && tma) stage1d_kernel<0, true><<<ntiles, NT1, 0, st>>>(probs, times, tiles, tb, sst, sn, out, m);
  else if (stage == 0) stage1d_kernel<0, false><<<ntiles, NT1, 0, st>>>(probs, times, tiles, tb, sst, sn, out, m);
  else if (tma) stage1d_kernel<1, true><<<ntiles, NT1, 0, st>>>(probs, times, tiles, tb, sst, sn, out, m);
  else stage1d_kernel<1, false><<<ntiles, NT1, 0, st>>>(probs, times, tiles, tb, sst, sn, out, m);
}

}  // namespace mdg
