// The dynamic shared memory that a kernel may be launched with.
#pragma once
#include <cuda_runtime.h>

namespace negf {

// What every kernel is allowed: 227 KB of a CTA less 4 KB for its static shared memory; the largest need is
// 221 KB (the Gauss-Jordan panels at n = 256).
constexpr size_t SMEM_LIMIT = 223 * 1024;

// Allow `smem` bytes.  The limit belongs to the kernel, not to a launch, so it is only ever set to the same
// value: a thread that sets it to what its own problem needs takes it from another thread's larger one,
// between that one's setting it and launching.
template <class Kernel>
inline bool allow_smem(Kernel* kernel, size_t smem) {
  return smem <= SMEM_LIMIT &&
         cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_LIMIT) == cudaSuccess;
}

}  // namespace negf
