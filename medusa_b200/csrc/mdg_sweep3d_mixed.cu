// Dendritic sweep, mixed precision: the MIX instantiations of the face kernels of
// mdg_sweep3d.cuh, in a translation unit of their own (MIXED2_FLAGS of medusa_b200/build.py).  As
// in the 2-D sweep the FP32 part of the work was bound by separate products and sums, rounded
// quotients and powf: 384 x 128 x 256 blast 5.87 -> 5.46 ms per step.
#include "mdg_sweep3d.cuh"

namespace mdg {

void launch_faces3_mixed(int stage, const FaceLaunch3 &f, const ProbDev *probs, ProbTime *times, const Grid3 &g,
                         StateSoA s, cudaStream_t st)
{
  if (stage == 0) launch_faces3<0, true>(f, probs, times, g, s, st);
  else launch_faces3<1, true>(f, probs, times, g, s, st);
}

}  // namespace mdg
