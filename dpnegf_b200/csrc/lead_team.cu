// The lead decimation and the lead adjoint with a thread-block cluster per work slot (see rgf_team.cu):
// products, triangular solves and elementwise passes are split over the cluster's CTAs, which each
// factorise their own copy of the LU panels.  Same operations per element, so bitwise equal results.
// n = 96 x 64 energies, Sigma and its parameter gradient: 16.2 -> 12.9 ms with two CTAs per slot.
#define NEGF_TEAM
#include "ls_item.cuh"
#include "lead_adjoint.cuh"
#include "team_launch.cuh"

namespace negf_team {

int ls_fit(size_t smem, int cl) { return negf::team_fit(ls_kernel, smem, cl); }
int ls_launch(const NegfLsProblem& p, size_t smem, int slots, int cl, cudaStream_t s) {
  return negf::team_launch(ls_kernel, p, smem, slots, cl, s);
}
int lead_adjoint_fit(size_t smem, int cl) { return negf::team_fit(lead_adjoint_kernel, smem, cl); }
int lead_adjoint_launch(const NegfLeadAdjProblem& p, size_t smem, int slots, int cl, cudaStream_t s) {
  return negf::team_launch(lead_adjoint_kernel, p, smem, slots, cl, s);
}

}  // namespace negf_team
