// Packing of the H/S blocks into the sweep's arena: one launch for every block.
//
// A device of K blocks has 9 K - 6 pieces (onsite, couplings, transposed copies); copying them one
// by one and testing the couplings for zero took about 10 launches per block, more than a
// single-energy sweep of a small junction.  Bound by the launches it replaces, not by bytes: the whole
// single-energy call of 8 blocks of 64 went from 3.18 to 1.71 ms.
#include "../../include/negf_b200.h"
#include "negf_common.cuh"

namespace NEGF_NS {

constexpr int PACK_THREADS = 256, PACK_PER_CTA = 4 * PACK_THREADS;

// CTA (x, y) copies entries x, x + gridDim.x, ... (in units of PACK_PER_CTA) of piece y.
__global__ void __launch_bounds__(PACK_THREADS) pack_kernel(const NegfPackPiece* pieces, cplx* arena, int32_t* nonzero) {
  const NegfPackPiece p = pieces[blockIdx.y];
  const cplx* src = reinterpret_cast<const cplx*>(p.src);
  cplx* dst = arena + p.dst;
  const int64_t count = (int64_t)p.rows * p.cols;
  bool nz = false;
  for (int64_t e0 = (int64_t)blockIdx.x * PACK_PER_CTA; e0 < count; e0 += (int64_t)gridDim.x * PACK_PER_CTA) {
#pragma unroll
    for (int s = 0; s < PACK_PER_CTA / PACK_THREADS; ++s) {
      const int64_t e = e0 + s * PACK_THREADS + threadIdx.x;
      if (e < count) {
        const int64_t i = e / p.cols, j = e % p.cols;
        cplx v = src[i * p.row_stride + j * p.col_stride];
        if (p.conj) v.y = -v.y;
        nz |= v.x != 0.0 || v.y != 0.0;
        dst[e] = v;
      }
    }
  }
  if (__syncthreads_or(nz) && threadIdx.x == 0) nonzero[blockIdx.y] = 1;
}

}  // namespace NEGF_NS

extern "C" int negf_pack_run(const NegfPackPiece* pieces, int32_t n_pieces, int64_t max_count, double* arena,
                             int32_t* nonzero, void* stream) {
  if (n_pieces < 0 || max_count < 0 || (n_pieces > 0 && (!pieces || !arena || !nonzero))) return NEGF_ERR_ARGUMENT;
  if (n_pieces == 0) return NEGF_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(nonzero, 0, (size_t)n_pieces * sizeof(int32_t), s) != cudaSuccess) return NEGF_ERR_CUDA;
  const int64_t chunks = (max_count + negf::PACK_PER_CTA - 1) / negf::PACK_PER_CTA;
  const unsigned gx = (unsigned)(chunks < 1 ? 1 : chunks < 64 ? chunks : 64);
  for (int32_t first = 0; first < n_pieces; first += 32768) {  // grid.y limit
    const int32_t n = n_pieces - first < 32768 ? n_pieces - first : 32768;
    negf::pack_kernel<<<dim3(gx, (unsigned)n), negf::PACK_THREADS, 0, s>>>(
        pieces + first, reinterpret_cast<negf::cplx*>(arena), nonzero + first);
  }
  return cudaGetLastError() == cudaSuccess ? NEGF_OK : NEGF_ERR_CUDA;
}
