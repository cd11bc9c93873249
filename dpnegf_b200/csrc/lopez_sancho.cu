// The C ABI of the lead decimation; the decimation itself is in ls_item.cuh.
#include "ls_item.cuh"
#include "team_launch.cuh"

namespace negf_team {
int ls_launch(const NegfLsProblem& p, size_t smem, int slots, int cl, cudaStream_t s);
int ls_fit(size_t smem, int cl);
}

namespace NEGF_NS {

size_t ls_smem_bytes(int max_n) { return lead_smem_bytes(max_n); }

}  // namespace NEGF_NS

extern "C" {

size_t negf_lopez_sancho_scratch_bytes(const NegfLsProblem* p) {
  if (!p || p->n_slots <= 0 || p->max_n <= 0) return 0;
  return negf::LS_SCRATCH_HEADER + (size_t)p->n_slots * negf::ls_slot_elems(*p) * sizeof(double2);
}

int negf_lopez_sancho_run(const NegfLsProblem* p, void* stream) { return negf_lopez_sancho_run_ctas(p, 0, stream); }

int negf_lopez_sancho_run_ctas(const NegfLsProblem* p, int32_t ctas, void* stream) {
  if (!p || !p->leads || !p->items || !p->arena || !p->status || !p->scratch) return NEGF_ERR_ARGUMENT;
  if (p->n_items <= 0) return NEGF_OK;
  if (p->max_n <= 0 || p->n_slots <= 0 || p->max_iter < 0) return NEGF_ERR_ARGUMENT;
  if (p->max_n > NEGF_MAX_BLOCK) return NEGF_ERR_UNSUPPORTED;
  if (p->scratch_bytes < negf_lopez_sancho_scratch_bytes(p)) return NEGF_ERR_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(p->scratch) & 255) != 0) return NEGF_ERR_ARGUMENT;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const size_t smem = negf::ls_smem_bytes(p->max_n);
  if (!negf::allow_smem(negf::ls_kernel, smem)) return NEGF_ERR_CUDA;
  const int grid = p->n_slots < p->n_items ? p->n_slots : p->n_items;
  const int cl =
      negf::team_choice(ctas, negf::ls_team_n(p->max_n), grid, [&](int c) { return negf_team::ls_fit(smem, c); });
  if (cl < 0) return NEGF_ERR_ARGUMENT;
  if (cudaMemsetAsync(p->scratch, 0, negf::LS_SCRATCH_HEADER, s) != cudaSuccess) return NEGF_ERR_CUDA;
  if (cl > 1) return negf_team::ls_launch(*p, smem, grid, cl, s);
  negf::ls_kernel<<<grid, negf::CTA_THREADS, smem, s>>>(*p);
  return cudaGetLastError() == cudaSuccess ? NEGF_OK : NEGF_ERR_CUDA;
}

}  // extern "C"
