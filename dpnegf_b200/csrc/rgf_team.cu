// The FP64 sweep with a thread-block cluster per work item, for launches with fewer items than the
// GPU has SMs: the cluster's CTAs split every block product by output tiles and every elementwise
// pass, repeat the in-register leaves of the inverse, and meet at cluster barriers.
#define NEGF_TEAM
#include "rgf_sweep.cuh"

namespace negf_team {

typedef void (*SweepKernel)(const NegfRgfProblem);

static SweepKernel team_kernel(int feat) {
  if (feat == FEAT_ADJOINT) return rgf_kernel<false, FEAT_ADJOINT>;
  if (feat == FEAT_LESSER) return rgf_kernel<false, FEAT_LESSER>;
  return rgf_kernel<false, FEAT_RETARDED>;
}

static void team_config(cudaLaunchConfig_t& c, cudaLaunchAttribute& a, size_t smem, int slots, int cl, cudaStream_t s) {
  a.id = cudaLaunchAttributeClusterDimension;
  a.val.clusterDim.x = (unsigned)cl;
  a.val.clusterDim.y = a.val.clusterDim.z = 1;
  c = cudaLaunchConfig_t{};
  c.gridDim = dim3((unsigned)(slots * cl));
  c.blockDim = dim3(CTA_THREADS);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &a;
  c.numAttrs = 1;
}

int rgf_team_fit(int feat, size_t smem, int cl) {
  cudaLaunchConfig_t c;
  cudaLaunchAttribute a;
  team_config(c, a, smem, 1, cl, nullptr);
  int n = 0;
  if (cudaFuncSetAttribute(team_kernel(feat), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, team_kernel(feat), &c) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int rgf_launch_team(int feat, const NegfRgfProblem& p, size_t smem, int slots, int cl, cudaStream_t s) {
  cudaLaunchConfig_t c;
  cudaLaunchAttribute a;
  team_config(c, a, smem, slots, cl, s);
  if (cudaFuncSetAttribute(team_kernel(feat), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return NEGF_ERR_CUDA;
  return cudaLaunchKernelEx(&c, team_kernel(feat), p) == cudaSuccess ? NEGF_OK : NEGF_ERR_CUDA;
}

}  // namespace negf_team
