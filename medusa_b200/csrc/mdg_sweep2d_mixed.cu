// 2-D sweep, mixed precision: the MIX instantiations of mdg_sweep2d.cuh, in a translation unit
// of their own because its multiplications and additions contract (MIXED2_FLAGS of
// medusa_b200/build.py), which the plain FP64 kernels must not.  Before, its FP32 products and
// sums were separate, every FP32 quotient and root was rounded correctly, and the
// two-rarefaction estimate called powf three times: at 2048^2 the FP32 pipe ran 20 of 46 M warp instructions of a direction-0 launch and the FP64 pipe 2.5 M.  With
// contraction, quot/root (mdg_hydro.cuh), pow_rarefaction and the next row's pencil on its way
// while a row is worked on: 1.89 -> 1.48 ms per step; error against 64 bits 5.7e-9 -> 5.4e-9
// (density, 700 x 500, 20 steps).
#include "mdg_sweep2d.cuh"

namespace mdg {

void launch_stage2d_mixed(int stage, const ProbDev *probs, ProbTime *times, const Tile *xtiles, int nxt,
                          const Tile *ytiles, int nyt, const Tables &tb, StateSoA sst, StateSoA sn, StateSoA acc,
                          StateSoA out, unsigned char *shock0, unsigned char *shock1, cudaStream_t st)
{
  launch_stage2d_as<true>(stage, probs, times, xtiles, nxt, ytiles, nyt, tb, sst, sn, acc, out, shock0, shock1, st);
}

}  // namespace mdg
