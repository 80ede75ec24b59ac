// The two forms of para_recon (mdg_recon.h) on the same seeded inputs, compared bit for bit:
// argv: seed, samples per grid.  Prints "grid samples flat declined different" per grid, then
// the same for div_by against the division operator.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "mdg_recon.h"
#include "mdg_tables.cuh"
using namespace mdg;
struct Row {
  const double *v;
  double operator()(int f) const { return v[f]; }
};
int main(int argc, char **argv)
{
  std::mt19937_64 rng(strtoull(argv[1], nullptr, 10));
  const long count = atol(argv[2]);
  auto u = [&] { return (rng() >> 11) * 0x1p-53; };
  // Cartesian and spherical; the smallest grid, ordinary and large ones, a domain in
  // centimetres, one that straddles the origin, one whose volumes leave the guarded range
  const struct { int n, sph; double len, x0; } grids[] = {
      {2, 0, 1.0, 0.0}, {2, 1, 1.0, 0.0}, {64, 0, 1.0, 0.0}, {64, 1, 1.0, 0.0}, {1024, 0, 1.0, 0.0}, {8192, 1, 1.0, 0.0},
      {8192, 0, 7.0e8, 0.0}, {8192, 1, 7.0e8, 0.0}, {4096, 0, 1.0, -0.5}, {64, 1, 1.0e-110, 0.0}};
  for (const auto &g : grids) {
    long flat = 0, declined = 0, differ = 0;
    const double dx = g.len / g.n;
    for (long t = 0; t < count; t++) {
      const int i = (int)(u() * (g.n + 2)) - 1;
      double al[3], be[3], ga[3], v[RC_NFIELDS];
      for (int k = 0; k < 3; k++) moments_closed(g.sph, g.x0, dx, i - 1 + k, al[k], be[k], ga[k]);
      rc_fields(al[0], al[1], al[2], be[0], be[1], be[2], ga[0], ga[1], ga[2], g.x0 + i * dx, g.x0 + (i + 1) * dx, v);
      const double size = pow(10.0, 40.0 * u() - 20.0), step = pow(10.0, -14.0 * u()), q = 2.0 * u() - 1.0;
      double w[3];
      switch (rng() % 6) {
        case 0: for (double &x : w) x = 2.0 * u() - 1.0; break;
        case 1: w[0] = q - step * u(); w[1] = q; w[2] = q + step * u(); break;
        case 2: w[0] = q - step * (1.0 + 1.0e-9 * u()); w[1] = q; w[2] = q + step; break;
        case 3: w[0] = q; w[1] = q + step; w[2] = q + 2.0 * step; break;
        case 4: for (double &x : w) x = 0.25 * (double)(rng() % 5) * (rng() % 2 ? 1.0 : -1.0); break;
        default: w[0] = u(); w[1] = w[0] * (1.0 + u()); w[2] = w[1] * pow(10.0, 8.0 * u()); break;
      }
      if (rng() % 500 == 0) w[rng() % 3] = (rng() % 2) ? INFINITY : NAN;
      if (rng() % 500 == 0) for (double &x : w) x *= 1.0e-280;
      for (double &x : w) x *= size;
      double l0, r0, l1, r1;
      para_recon_zone<double>(w[0], w[1], w[2], Row{v}, l0, r0);
      const bool ok = para_recon_fast(w[0], w[1], w[2], Row{v}, l1, r1);
      if ((w[1] - w[0]) * (w[2] - w[1]) <= 0.0) flat++;
      if (!ok) declined++;
      else if (memcmp(&l0, &l1, 8) || memcmp(&r0, &r1, 8)) differ++;
    }
    printf("%d/%d/%g/%g %ld %ld %ld %ld\n", g.n, g.sph, g.len, g.x0, count, flat, declined, differ);
  }
  long differ = 0;
  for (long t = 0; t < 10 * count; t++) {
    double b = (1.0 + u()) * pow(2.0, (int)(400.0 * u()) - 200), a = (1.0 + u()) * pow(2.0, (int)(400.0 * u()) - 200);
    if (t % 3 == 1) a = b * (double)(rng() % 1000 + 1);
    if (t % 3 == 2) {   // divisors next below a power of two
      int64_t m;
      memcpy(&m, &b, 8);
      m = (m | 0x000fffffffffffffLL) - (int64_t)(rng() % 64);
      memcpy(&b, &m, 8);
    }
    if (div_by(a, b, 1.0 / b) != a / b) differ++;
  }
  printf("div %ld 0 0 %ld\n", 10 * count, differ);
  return 0;
}
