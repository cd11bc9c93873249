// The FP64 sweep with a thread-block cluster per work item, for launches with fewer items than the
// GPU has SMs: the cluster's CTAs split every block product by output tiles and every elementwise
// pass, repeat the in-register leaves of the inverse, and meet at cluster barriers.  Bound by the
// repeated leaves (57 us per 64 rows) and the products' largest share.  One CTA per item -> a team:
// b = 100..130 x 18 blocks x 50 energies 16.5 -> 10.8 ms (two CTAs), lesser b = 128 x 6 x 64
// 12.0 -> 8.2 (two), one energy of b = 64 x 8 with all blocks 3.34 -> 3.18 (two; its calls dominate).
#define NEGF_TEAM
#include "rgf_sweep.cuh"
#include "team_launch.cuh"

namespace negf_team {

typedef void (*SweepKernel)(const NegfRgfProblem);

static SweepKernel team_kernel(int feat) {
  if (feat == FEAT_ADJOINT) return rgf_kernel<false, FEAT_ADJOINT>;
  if (feat == FEAT_LESSER) return rgf_kernel<false, FEAT_LESSER>;
  return rgf_kernel<false, FEAT_RETARDED>;
}

int rgf_team_fit(int feat, size_t smem, int cl) { return negf::team_fit(team_kernel(feat), smem, cl); }

int rgf_launch_team(int feat, const NegfRgfProblem& p, size_t smem, int slots, int cl, cudaStream_t s) {
  return negf::team_launch(team_kernel(feat), p, smem, slots, cl, s);
}

}  // namespace negf_team
