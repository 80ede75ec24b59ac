// 2-D sweep: the plain FP64 launches (compiled without multiply-add contraction) and the tile
// rule of both precisions.
#include "mdg_sweep2d.cuh"

namespace mdg {

// Rows per tile.  A tile marches down its rows one after the other, so its time is that of
// its rows (and of what it does once: two more reconstructed rows in direction 0, the
// column tables in direction 1), and a row takes a nearly fixed time while few CTAs share
// an SM (a chain of dependent FP64 operations) and a time that grows with them once four
// do.  Measured on a B200 when the rule was made, plain FP64 with the dividing reconstruction: a
// direction-0 row 6.5 us alone on its SM and 11 us beside three others, a direction-1 row 13 us
// and 14 us; the kernels are faster since, and the rule was not measured again.  The count
// with the smallest modelled time is taken: full-size grids keep long tiles (2048^2: 32 and 15
// rows), small ones are cut until the chip is full -- 512^2 with 32 and 16 rows gave 64 and 160
// CTAs for 592 places, and a step took 1.0 ms (0.268 ms now, 296 and 515 CTAs).  The mixed sweep,
// whose kernels hold 3 CTAs per SM, takes the same tiles.
int tile_rows_2d(int dir, const int *n1, const int *n2, int n, int num_sms)
{
  const int most = dir ? TIY2 : TIX2, cols = dir ? TJY2 : NTX2;
  const double alone = dir ? 13.0 : 6.5, shared = dir ? 3.5 : 2.75, once = dir ? 0.4 : 2.0;
  const int per_sm = dir ? MDG_YMINB : MDG_XMINB;
  const int sms = num_sms > 0 ? num_sms : 148;
  int best = most;
  double tbest = 0.0;
  for (int rows = most; rows >= 1; rows--) {
    long long tiles = 0;
    for (int m = 0; m < n; m++) tiles += (long long)((n1[m] + rows - 1) / rows) * ((n2[m] + cols - 1) / cols);
    const long long wave = (long long)per_sm * sms, full = tiles / wave, rest = tiles - full * wave;
    auto row_time = [&](long long k) { return k <= 0 ? 0.0 : (k * shared > alone ? k * shared : alone); };
    const double t = (rows + once) * ((double)full * row_time(per_sm) + row_time((rest + sms - 1) / sms));
    if (rows == most || t < 0.97 * tbest) {
      best = rows;
      tbest = t;
    }
  }
  return best;
}

void launch_stage2d_mixed(int stage, const ProbDev *probs, ProbTime *times, const Tile *xtiles, int nxt,
                          const Tile *ytiles, int nyt, const Tables &tb, StateSoA sst, StateSoA sn, StateSoA acc,
                          StateSoA out, unsigned char *shock0, unsigned char *shock1, cudaStream_t st);

void launch_stage2d(int stage, bool mixed, const ProbDev *probs, ProbTime *times, const Tile *xtiles, int nxt,
                    const Tile *ytiles, int nyt, const Tables &tb, StateSoA sst, StateSoA sn, StateSoA acc,
                    StateSoA out, unsigned char *shock0, unsigned char *shock1, cudaStream_t st)
{
  if (nxt <= 0 || nyt <= 0) return;
  if (mixed)
    launch_stage2d_mixed(stage, probs, times, xtiles, nxt, ytiles, nyt, tb, sst, sn, acc, out, shock0, shock1, st);
  else
    launch_stage2d_as<false>(stage, probs, times, xtiles, nxt, ytiles, nyt, tb, sst, sn, acc, out, shock0, shock1, st);
}

}  // namespace mdg
