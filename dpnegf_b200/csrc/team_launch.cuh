// Host side of the cluster launches.
#pragma once
#include <cuda_runtime.h>
#include "../../include/negf_b200.h"
#include "smem_limit.cuh"
#include "team_rule.cuh"

namespace negf {

// team_rule on the current GPU.
template <class Fit>
inline int team_ctas(int n, int slots, Fit fit) {
  int dev = 0, sms = 0;
  if (n <= 32 || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 1;
  return team_rule(n, slots, sms, fit);
}

// The same for a caller's choice: 0 the rule, 1, 2, 4 or 8 CTAs per slot whatever the slots (clusters
// that do not fit together wait for each other); -1 when the GPU cannot run it.
template <class Fit>
inline int team_choice(int ctas, int n, int slots, Fit fit) {
  if (ctas == 0) return team_ctas(n, slots, fit);
  if (ctas == 1) return 1;
  return (ctas == 2 || ctas == 4 || ctas == 8) && fit(ctas) > 0 ? ctas : -1;
}

inline void team_config(cudaLaunchConfig_t& c, cudaLaunchAttribute& a, size_t smem, int slots, int cl, cudaStream_t s) {
  a.id = cudaLaunchAttributeClusterDimension;
  a.val.clusterDim.x = (unsigned)cl;
  a.val.clusterDim.y = a.val.clusterDim.z = 1;
  c = cudaLaunchConfig_t{};
  c.gridDim = dim3((unsigned)(slots * cl));
  c.blockDim = dim3(256);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &a;
  c.numAttrs = 1;
}

// Clusters of `cl` CTAs that run at once; 0 when the GPU cannot run them.
template <class Problem>
inline int team_fit(void (*kernel)(const Problem), size_t smem, int cl) {
  cudaLaunchConfig_t c;
  cudaLaunchAttribute a;
  team_config(c, a, smem, 1, cl, nullptr);
  int n = 0;
  if (!allow_smem(kernel, smem) || cudaOccupancyMaxActiveClusters(&n, kernel, &c) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

template <class Problem>
inline int team_launch(void (*kernel)(const Problem), const Problem& p, size_t smem, int slots, int cl, cudaStream_t s) {
  cudaLaunchConfig_t c;
  cudaLaunchAttribute a;
  team_config(c, a, smem, slots, cl, s);
  if (!allow_smem(kernel, smem)) return NEGF_ERR_CUDA;
  return cudaLaunchKernelEx(&c, kernel, p) == cudaSuccess ? NEGF_OK : NEGF_ERR_CUDA;
}

}  // namespace negf
