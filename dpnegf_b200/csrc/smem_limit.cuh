// The dynamic shared memory that a kernel may be launched with.
#pragma once
#include <cuda_runtime.h>

namespace negf {

// Allow `smem` bytes.  The limit belongs to the kernel, not to a launch, so it is only ever set to all that
// the GPU has beside the kernel's static shared memory: a thread that sets it to what its own problem needs
// takes it from another thread's larger one, between that one's setting it and launching.
template <class Kernel>
inline bool allow_smem(Kernel* kernel, size_t smem) {
  cudaFuncAttributes a;
  int dev = 0, most = 0;
  if (cudaFuncGetAttributes(&a, kernel) != cudaSuccess) return false;
  if ((size_t)a.maxDynamicSharedSizeBytes >= smem) return true;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return false;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes) ==
         cudaSuccess;
}

}  // namespace negf
