// Product chains around the sweep and the decimation (sm_100a, FP64 tensor cores):
//
//   negf_gamma_sum_run      out = sum_i w_i Re(G_i[:, c0:c0+k] Gamma_i G_i[:, c0:c0+k]^H)
//                           the non-equilibrium density matrix of Ozaki.integrate
//                           (negf/density.py:183-195, DM_neq = sum w (G Gamma_R G^H).real (f_R - f_L))
//   negf_lead_adjoint_run   dL/d(H, H01, S, S01, H_DL, S_DL) of a lead's self-energies through the
//                           converged decimation fixed point (the implicit-function adjoint of
//                           g_s = (zS - H - tau g_s tau')^-1, the relation the reference's residual
//                           check tests, negf/surface_green.py:142-145)
//
// Both are batched over energies and use the CTA tile GEMM of the sweep (DMMA, Gauss/3M complex
// products, as the sweep: no iteration here feeds rounding back) and the pivoted LU of the
// decimation.  Sums over energies run in a fixed order, so
// results are bitwise reproducible.
#include "../../include/negf_b200.h"
#include "lead_adjoint.cuh"
#include "team_launch.cuh"

namespace negf_team {
int lead_adjoint_launch(const NegfLeadAdjProblem& p, size_t smem, int slots, int cl, cudaStream_t s);
int lead_adjoint_fit(size_t smem, int cl);
}

namespace NEGF_NS {

// ---------------------------------------------------------------------------------------------
// Weighted G Gamma G^H sum.  Stage 1 (one CTA per energy): T_i = w_i G_i[:, c0:] Gamma_i and a
// copy of G_i[:, c0:], side by side as the column blocks of two n x (n_items k) matrices.
// Stage 2: out = Re(T_stack G_stack^H), one GEMM over every energy.  Its k-loop is split into
// up to GS_MAX_SPLIT contiguous ranges so that the output tiles times the splits fill the GPU
// (a 256 x 256 output is only 16 tiles); each (tile, range) CTA writes the real part of its
// partial product, and stage 3 sums the ranges in range order, so the result does not depend
// on scheduling.

constexpr size_t PROD_ALIGN = 256;
constexpr int GS_MAX_SPLIT = 16;

inline size_t round_up(size_t b) { return (b + PROD_ALIGN - 1) & ~(PROD_ALIGN - 1); }

inline size_t gamma_stack_bytes(const NegfGammaSum& p) {
  return round_up((size_t)p.n * (size_t)p.n_items * (size_t)p.k * sizeof(cplx));
}

inline size_t gamma_part_bytes(const NegfGammaSum& p) {
  return round_up((size_t)GS_MAX_SPLIT * p.n * p.n * sizeof(double));
}

// k-range length of stage 2 for `split` ranges: a multiple of the 16-deep k slab.
inline int64_t gamma_split_len(int64_t K, int split) { return ((K + split - 1) / split + 15) / 16 * 16; }

__global__ void __launch_bounds__(CTA_THREADS, 1) gamma_stack_kernel(const NegfGammaSum P, cplx* Tst, cplx* Gst) {
  char* const smem_raw = negf_smem;
  cplx* smem = reinterpret_cast<cplx*>(smem_raw);
  const int64_t K = (int64_t)P.n_items * P.k;
  for (int i = blockIdx.x; i < P.n_items; i += gridDim.x) {
    const cplx* G = reinterpret_cast<const cplx*>(P.g) + (int64_t)i * P.g_stride + P.c0;
    const cplx* Gam = reinterpret_cast<const cplx*>(P.gamma) + (int64_t)i * P.gamma_stride;
    gemm_ls<OP_N, OP_N, true>(smem, P.n, P.k, P.k, G, P.ldg, Gam, P.ldgam, Tst + (int64_t)i * P.k, K, nullptr, 0,
                        cmk(P.w[i], 0.0));
    for (int64_t e = threadIdx.x; e < (int64_t)P.n * P.k; e += CTA_THREADS) {
      const int64_t r = e / P.k, c = e % P.k;
      Gst[r * K + (int64_t)i * P.k + c] = G[r * P.ldg + c];
    }
    __syncthreads();
  }
}

struct EpiRealOut {
  double* out;
  int64_t ld;
  int m0, n0;
  NEGF_DEV void operator()(int m, int n, cplx v) const { out[(int64_t)(m0 + m) * ld + n0 + n] = v.x; }
};

// Stage 2: CTA (x, y, z) multiplies output tile (y, x) over k-range z into part[z].
__global__ void __launch_bounds__(CTA_THREADS, 1) gamma_reduce_kernel(const NegfGammaSum P, const cplx* Tst,
                                                                      const cplx* Gst, double* part,
                                                                      int64_t klen) {
  char* const smem_raw = negf_smem;
  cplx* smem = reinterpret_cast<cplx*>(smem_raw);
  const int64_t K = (int64_t)P.n_items * P.k;
  const int m0 = blockIdx.y * GT_M, n0 = blockIdx.x * GT_N;
  const int64_t k0 = (int64_t)blockIdx.z * klen;
  const int M = min(GT_M, P.n - m0), N = min(GT_N, P.n - n0);
  const int Kz = (int)(k0 < K ? (K - k0 < klen ? K - k0 : klen) : 0);
  double* out = part + (size_t)blockIdx.z * P.n * P.n;
  if (Kz == 0) {  // an empty range still writes its (zero) partial tile
    for (int e = threadIdx.x; e < M * N; e += CTA_THREADS) out[(int64_t)(m0 + e / N) * P.n + n0 + e % N] = 0.0;
    return;
  }
  GemmArgs g = gemm_args(M, N, Kz, Tst + (int64_t)m0 * K + k0, K, Gst + (int64_t)n0 * K + k0, K, nullptr, 0);
  cta_gemm_epi<OP_N, OP_C, true, true>(g, EpiRealOut{out, P.n, m0, n0});
}

// Stage 3: out = sum of the partial outputs in range order.
__global__ void gamma_sum_parts_kernel(double* out, const double* part, int64_t n2, int split) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n2; e += (int64_t)gridDim.x * blockDim.x) {
    double s = part[e];
    for (int z = 1; z < split; ++z) s += part[(size_t)z * n2 + e];
    out[e] = s;
  }
}

// grad[e] = sum over slots, in slot order, of the slots' accumulators.
__global__ void lead_adjoint_sum_kernel(const NegfLeadAdjProblem P, int slots) {
  const int64_t n2 = (int64_t)P.lead.n * P.lead.n;
  const int64_t total = la_grad_elems(P);
  const size_t mn = (size_t)la_max_n(P.lead), mn2 = mn * mn;
  const cplx* base = reinterpret_cast<const cplx*>(P.scratch);
  cplx* out = reinterpret_cast<cplx*>(P.grad);
  const size_t stride = la_slot_elems(P);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int r;
    int64_t off;
    if (e < 4 * n2) { r = (int)(e / n2); off = e % n2; }
    else { const int64_t ncb = (int64_t)P.lead.nc * P.lead.b; r = 4 + (int)((e - 4 * n2) / ncb); off = (e - 4 * n2) % ncb; }
    cplx s = cmk(0.0, 0.0);
    for (int k = 0; k < slots; ++k) s = cadd(s, base[(size_t)k * stride + r * mn2 + off]);
    out[e] = s;
  }
}

static int sm_count_or(int fallback) {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fallback;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return fallback;
  return n > 0 ? n : fallback;
}

}  // namespace NEGF_NS

extern "C" {

size_t negf_gamma_sum_scratch_bytes(const NegfGammaSum* p) {
  if (!p || p->n <= 0 || p->k <= 0 || p->n_items <= 0) return 0;
  return 2 * negf::gamma_stack_bytes(*p) + negf::gamma_part_bytes(*p);
}

int negf_gamma_sum_run(const NegfGammaSum* p, void* stream) {
  if (!p || !p->g || !p->gamma || !p->w || !p->out) return NEGF_ERR_ARGUMENT;
  if (p->n <= 0 || p->k <= 0 || p->n_items < 0 || p->c0 < 0 || p->ldg < p->c0 + p->k || p->ldgam < p->k)
    return NEGF_ERR_ARGUMENT;
  if ((int64_t)p->n_items * p->k > 0x7fffffff) return NEGF_ERR_UNSUPPORTED;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (p->n_items == 0)
    return cudaMemsetAsync(p->out, 0, (size_t)p->n * p->n * sizeof(double), s) == cudaSuccess ? NEGF_OK : NEGF_ERR_CUDA;
  if (!p->scratch || p->scratch_bytes < negf_gamma_sum_scratch_bytes(p)) return NEGF_ERR_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(p->scratch) & 255) != 0) return NEGF_ERR_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(p->g) & 15) || (reinterpret_cast<uintptr_t>(p->gamma) & 15)) return NEGF_ERR_ARGUMENT;
  negf::cplx* Tst = reinterpret_cast<negf::cplx*>(p->scratch);
  negf::cplx* Gst = reinterpret_cast<negf::cplx*>(reinterpret_cast<char*>(p->scratch) + negf::gamma_stack_bytes(*p));
  const int smem = negf::GEMM_SMEM_BYTES;
  if (!negf::allow_smem(negf::gamma_stack_kernel, smem) || !negf::allow_smem(negf::gamma_reduce_kernel, smem))
    return NEGF_ERR_CUDA;
  const int sms = negf::sm_count_or(148);
  const int grid1 = p->n_items < sms ? p->n_items : sms;
  negf::gamma_stack_kernel<<<grid1, negf::CTA_THREADS, smem, s>>>(*p, Tst, Gst);
  double* part = reinterpret_cast<double*>(reinterpret_cast<char*>(p->scratch) + 2 * negf::gamma_stack_bytes(*p));
  const int tiles = (p->n + negf::GT_M - 1) / negf::GT_M;
  const int64_t K = (int64_t)p->n_items * p->k;
  int split = (2 * sms + tiles * tiles - 1) / (tiles * tiles);  // about two CTAs per SM
  if (split > negf::GS_MAX_SPLIT) split = negf::GS_MAX_SPLIT;
  if ((int64_t)split > (K + 255) / 256) split = (int)((K + 255) / 256);  // keep ranges >= 256 deep
  if (split < 1) split = 1;
  const int64_t klen = negf::gamma_split_len(K, split);
  negf::gamma_reduce_kernel<<<dim3(tiles, tiles, split), negf::CTA_THREADS, smem, s>>>(*p, Tst, Gst, part, klen);
  const int64_t n2 = (int64_t)p->n * p->n;
  const int rgrid = (int)((n2 + 255) / 256 < 1024 ? (n2 + 255) / 256 : 1024);
  negf::gamma_sum_parts_kernel<<<rgrid, 256, 0, s>>>(p->out, part, n2, split);
  return cudaGetLastError() == cudaSuccess ? NEGF_OK : NEGF_ERR_CUDA;
}

size_t negf_lead_adjoint_scratch_bytes(const NegfLeadAdjProblem* p) {
  if (!p || p->n_slots <= 0 || p->lead.n <= 0) return 0;
  return (size_t)p->n_slots * negf::la_slot_elems(*p) * sizeof(double2);
}

int negf_lead_adjoint_run(const NegfLeadAdjProblem* p, void* stream) { return negf_lead_adjoint_run_ctas(p, 0, stream); }

int negf_lead_adjoint_run_ctas(const NegfLeadAdjProblem* p, int32_t ctas, void* stream) {
  if (!p || !p->arena || !p->items || !p->grad || !p->status || !p->scratch) return NEGF_ERR_ARGUMENT;
  const NegfLead& ld = p->lead;
  if (ld.n <= 0 || p->n_slots <= 0 || p->max_iter < 0 || p->form < 0 || p->form > 2) return NEGF_ERR_ARGUMENT;
  if (ld.n > NEGF_MAX_BLOCK || ld.nc > NEGF_MAX_BLOCK) return NEGF_ERR_UNSUPPORTED;
  if (p->form == 0 && (ld.nc <= 0 || ld.b <= 0 || ld.b > ld.n || ld.hdl < 0 || ld.sdl < 0)) return NEGF_ERR_ARGUMENT;
  if (p->scratch_bytes < negf_lead_adjoint_scratch_bytes(p)) return NEGF_ERR_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(p->scratch) & 255) != 0) return NEGF_ERR_ARGUMENT;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (p->n_items <= 0)
    return cudaMemsetAsync(p->grad, 0, (size_t)negf::la_grad_elems(*p) * sizeof(double2), s) == cudaSuccess
               ? NEGF_OK : NEGF_ERR_CUDA;
  const size_t smem = negf::lead_smem_bytes(negf::la_max_n(ld));
  if (!negf::allow_smem(negf::lead_adjoint_kernel, smem)) return NEGF_ERR_CUDA;
  const int grid = p->n_slots < p->n_items ? p->n_slots : p->n_items;
  const int cl = negf::team_choice(ctas, ld.n, grid, [&](int c) { return negf_team::lead_adjoint_fit(smem, c); });
  if (cl < 0) return NEGF_ERR_ARGUMENT;
  if (cl > 1) {
    const int st = negf_team::lead_adjoint_launch(*p, smem, grid, cl, s);
    if (st != NEGF_OK) return st;
  } else {
    negf::lead_adjoint_kernel<<<grid, negf::CTA_THREADS, smem, s>>>(*p);
  }
  const int64_t total = negf::la_grad_elems(*p);
  const int rgrid = (int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
  negf::lead_adjoint_sum_kernel<<<rgrid, 256, 0, s>>>(*p, grid);
  return cudaGetLastError() == cudaSuccess ? NEGF_OK : NEGF_ERR_CUDA;
}

}  // extern "C"
