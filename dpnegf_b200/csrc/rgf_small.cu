// The FP64 sweep for blocks of up to 32 and more items than SMs: two-warp CTAs with 32 x 32 tiles,
// three to an SM.  A small block's steps are chains of short latencies (a 2 x 2 product took as long
// as a 32 x 32 one); three items per SM overlap them (shared memory sets the three: 62 KB of ring).
// Whole T + DOS calls, one 256-thread CTA per SM -> three small ones: b = 2 x 10 blocks x 1000
// energies 1.90 -> 1.15 ms, b = 8 x 20 x 1500 6.33 -> 3.67, b = 16 x 20 x 200 1.75 -> 1.33,
// b = 32 x 20 x 300 4.27 -> 2.70, b = 32 x 20 x 1000 9.56 -> 7.89.
#define NEGF_SMALL
#include "rgf_sweep.cuh"

namespace negf_small {

int rgf_launch_small(int feat, const NegfRgfProblem& p, int grid, cudaStream_t s) {
  const size_t smem = rgf_smem_bytes(32, false);
  if (feat == FEAT_ADJOINT) return rgf_launch_impl<false, FEAT_ADJOINT>(p, smem, grid, s);
  if (feat == FEAT_LESSER) return rgf_launch_impl<false, FEAT_LESSER>(p, smem, grid, s);
  return rgf_launch_impl<false, FEAT_RETARDED>(p, smem, grid, s);
}

}  // namespace negf_small
