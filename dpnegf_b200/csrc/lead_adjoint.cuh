// The lead adjoint of products.cu, compiled for one CTA and for a cluster per work slot.
#pragma once
#include "../../include/negf_b200.h"
#include "lead_forms.cuh"

namespace NEGF_NS {

// ---------------------------------------------------------------------------------------------
// Lead adjoint.  Per energy (z = E + i eta, tau = z S01 - H01, tau' = z S01^H - H01^H, g = g_s):
//   V = dL/dg from Sigma(g):  form 0  Sigma = L g[:b,:b] R,  L = E S_DL - H_DL, R = E S_DL^H - H_DL^H
//                                      V[:b,:b] = L^H Gs R^H,  dL/dL = Gs R^H g_b^H,  dL/dR = g_b^H L^H Gs
//                             form 1  Sigma = g^-1:           V = -g^-H Gs g^-H
//                             form 2  Sigma = E S - H - g^-1: V = +g^-H Gs g^-H, dS += conj(E) Gs, dH -= Gs
//   Lambda = V + P^H Lambda Q^H with P = g tau, Q = tau' g, by doubling
//            (Lambda += P^H Lambda Q^H, P <- P^2, Q <- Q^2 until max|P| max|Q| < tol)
//   F = (zS - H - tau g tau')^-1, dW = -F^H Lambda F^H
//   dS += conj(z) dW, dH -= dW, dtau = -dW (g tau')^H, dtau' = -(tau g)^H dW,
//   dS01 += conj(z) dtau + z dtau'^H, dH01 -= dtau + dtau'^H
// (PyTorch's convention: the gradient of a real loss w.r.t. a complex tensor is dL/d conj(x)).
// Energies go to the CTAs round-robin; each CTA sums its energies' contributions in its own slot,
// and a second kernel sums the slots in slot order.

// The product of one tile and one k = 8 step (the leads of up to 8, a few dozen products per energy): no
// ring, and no MMAs for the empty half of the 16-deep slab, which is half of them.  The drifting form's
// larger start-up had made the lead adjoint of such leads 3-8 % slower than the form before it.  Lead
// adjoint, 148 energies: n = 1 201 -> 143 us, n = 8 245 -> 176 (191 and 232 before the drifting form).
// Skipping the empty half inside the tile GEMM's loop instead cost the large products 1-3 %, and the same
// choice in the decimation 5 % of its steps at n = 33..64.
template <int OPA, int OPB, bool G3>
__device__ __noinline__ void cta_gemm_thin(const GemmArgs& gr) {
  const GemmArgs g = gr;
  cplx *sA = smem_cplx(), *sB = sA + GT_TILE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 32, wn = ((warp + 2 * (warp >> 2)) & 3) * 16;  // as the drifting form
  typedef typename std::conditional<OPA == OP_C, AIdxOpC, AIdxOp0>::type AI;
  typedef typename std::conditional<OPB == OP_C, BIdxOpC, BIdxOp0>::type BI;
  if (team_rank() == 0) {
    __syncthreads();  // whatever used this memory before is done with it
    load_a_tile<OPA>(sA, g, 0, 0, tid);
    load_b_tile<OPB>(sB, g, 0, 0, tid);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (wm < g.M && wn < g.N) {
      Acc3M acc;
      acc.zero();
      warp_mma_3m<(OPA != OP_N), (OPB != OP_N), G3>(acc, sA, sB, 1, wm, wn, lane, AI(), BI());
      const EpiStore epi{g};
      acc_foreach<G3>(acc, wm, wn, lane, [&](int m, int n, cplx v) {
        if (m < g.M && n < g.N) epi(m, n, v);
      });
    }
  }
  team_sync();
}

// gemm_ls with Gauss/3M products, thin where it can be.
template <int OPA, int OPB>
NEGF_DEV void gemm_la(cplx* smem, int M, int N, int K, const cplx* A, int64_t lda, const cplx* B, int64_t ldb, cplx* C,
                      int64_t ldc, const cplx* D = nullptr, int64_t ldd = 0, cplx alpha = cmk(1.0, 0.0)) {
  if (K > 8 || M > GT_M || N > GT_N) {
    gemm_ls<OPA, OPB, true>(smem, M, N, K, A, lda, B, ldb, C, ldc, D, ldd, alpha);
    return;
  }
  GemmArgs g = gemm_args(M, N, K, A, lda, B, ldb, C, ldc);
  g.alpha = alpha;
  if (D) { g.D = D; g.ldd = ldd; g.beta = cmk(1.0, 0.0); g.use_d = true; }
  cta_gemm_thin<OPA, OPB, true>(g);
}

constexpr int LA_NACC = 6, LA_NWORK = 12;

__host__ __device__ inline int la_max_n(const NegfLead& ld) { return ld.nc > ld.n ? ld.nc : ld.n; }

__host__ __device__ inline size_t la_slot_elems(const NegfLeadAdjProblem& p) {
  const size_t mn = (size_t)la_max_n(p.lead);
  return ((LA_NACC + LA_NWORK) * mn * mn + 15) & ~(size_t)15;
}

__host__ __device__ inline int64_t la_grad_elems(const NegfLeadAdjProblem& p) {
  const int64_t n = p.lead.n, ncb = p.form == 0 ? (int64_t)p.lead.nc * p.lead.b : 0;
  return 4 * n * n + 2 * ncb;
}

NEGF_DEV void la_item(const NegfLeadAdjProblem& P, int idx, cplx* slot, char* smem_raw, double* red) {
  cplx* smem = reinterpret_cast<cplx*>(smem_raw);
  const NegfLead ld = P.lead;
  const int n = ld.n;
  const int64_t n2 = (int64_t)n * n;
  const size_t mn = (size_t)la_max_n(ld), mn2 = mn * mn;
  const NegfLeadAdjItem it = P.items[idx];
  const cplx* ar = reinterpret_cast<const cplx*>(P.arena);
  const cplx *H = ar + ld.h, *S = ar + ld.s, *H01 = ar + ld.h01, *S01 = ar + ld.s01;
  const cplx* g = reinterpret_cast<const cplx*>(it.gs);
  const cplx* Gs = reinterpret_cast<const cplx*>(it.gsig);
  const cplx E = cmk(it.e_re, it.e_im);
  const cplx z = cmk(it.e_re, it.e_im + P.eta);
  const cplx ONE = cmk(1.0, 0.0), MONE = cmk(-1.0, 0.0);
  cplx* acc[LA_NACC];
  for (int r = 0; r < LA_NACC; ++r) acc[r] = slot + r * mn2;
  cplx* w_[LA_NWORK];
  for (int r = 0; r < LA_NWORK; ++r) w_[r] = slot + (LA_NACC + r) * mn2;
  cplx *lam = w_[0], *Pm = w_[1], *Qm = w_[2], *P2 = w_[3], *Q2 = w_[4], *T1 = w_[5];
  cplx *tau = w_[6], *taup = w_[7], *Y1 = w_[8], *W = w_[9], *F = w_[10], *gW = w_[11];
  int bad = 0;

  // ---- V = dL/dg into lam
  for (int64_t e = team_tid(); e < n2; e += team_threads()) lam[e] = cmk(0.0, 0.0);
  team_sync();
  if (P.form == 0) {
    const int nc = ld.nc, b = ld.b;
    const cplx *hdl = ar + ld.hdl, *sdl = ar + ld.sdl;
    cplx *Lm = Pm, *Rm = Qm, *T2 = P2, *gL = Q2, *gR = Y1;
    for (int e = team_tid(); e < nc * b; e += team_threads()) Lm[e] = csub(cmul(E, sdl[e]), hdl[e]);
    team_sync();
    form_eS_minus_h_herm(Rm, hdl, sdl, E, b, nc);                       // b x nc
    gemm_la<OP_C, OP_N>(smem, b, nc, nc, Lm, b, Gs, nc, T1, nc);        // L^H Gs       (b x nc)
    gemm_la<OP_N, OP_C>(smem, b, b, nc, T1, nc, Rm, nc, lam, n);        // V[:b,:b]
    gemm_la<OP_N, OP_C>(smem, nc, b, nc, Gs, nc, Rm, nc, T2, b);        // Gs R^H       (nc x b)
    gemm_la<OP_N, OP_C>(smem, nc, b, b, T2, b, g, n, gL, b);            // dL/dL        (nc x b)
    gemm_la<OP_C, OP_N>(smem, b, nc, b, g, n, T1, nc, gR, nc);          // dL/dR        (b x nc)
    const cplx Ec = cconj(E);
    for (int e = team_tid(); e < nc * b; e += team_threads()) {
      const int i = e / b, j = e % b;
      const cplx l = gL[e], rH = cconj(gR[(int64_t)j * nc + i]);
      acc[4][e] = csub(acc[4][e], cadd(l, rH));                          // H_DL
      acc[5][e] = cadd(acc[5][e], cadd(cmul(Ec, l), cmul(E, rH)));      // S_DL
    }
    team_sync();
  } else {
    for (int64_t e = team_tid(); e < n2; e += team_threads()) F[e] = g[e];
    team_sync();
    bad |= cta_lu_inverse(F, W, n, smem_raw);                           // W = g^-1
    gemm_la<OP_C, OP_N>(smem, n, n, n, W, n, Gs, n, T1, n);             // g^-H Gs
    gemm_la<OP_N, OP_C>(smem, n, n, n, T1, n, W, n, lam, n, nullptr, 0, P.form == 1 ? MONE : ONE);
    if (P.form == 2) {
      const cplx Ec = cconj(E);
      for (int64_t e = team_tid(); e < n2; e += team_threads()) {
        acc[0][e] = csub(acc[0][e], Gs[e]);
        acc[2][e] = cadd(acc[2][e], cmul(Ec, Gs[e]));
      }
      team_sync();
    }
  }

  // ---- Lambda by doubling
  cta_shift_form<true>(tau, H01, S01, z, MONE, (int)n2, smem);                // z S01 - H01
  form_eS_minus_h_herm(taup, H01, S01, z, n, n);                        // z S01^H - H01^H
  gemm_la<OP_N, OP_N>(smem, n, n, n, g, n, tau, n, Pm, n);              // P = g tau
  gemm_la<OP_N, OP_N>(smem, n, n, n, taup, n, g, n, Qm, n);             // Q = tau' g
  int steps = 0;
  bool finite = true;
  for (int s = 0; s < P.max_iter; ++s) {
    steps = s + 1;
    gemm_la<OP_C, OP_N>(smem, n, n, n, Pm, n, lam, n, T1, n);           // P^H Lambda
    gemm_la<OP_N, OP_C>(smem, n, n, n, T1, n, Qm, n, lam, n, lam, n);   // Lambda += ... Q^H
    gemm_la<OP_N, OP_N>(smem, n, n, n, Pm, n, Pm, n, P2, n);
    gemm_la<OP_N, OP_N>(smem, n, n, n, Qm, n, Qm, n, Q2, n);
    cplx* t = Pm; Pm = P2; P2 = t;
    t = Qm; Qm = Q2; Q2 = t;
    double mp = 0.0, mq = 0.0;
    for (int64_t e = team_tid(); e < n2; e += team_threads()) {
      const double a = hypot(Pm[e].x, Pm[e].y), c = hypot(Qm[e].x, Qm[e].y);
      mp = (a == a) ? fmax(mp, a) : INFINITY;
      mq = (c == c) ? fmax(mq, c) : INFINITY;
    }
    mp = team_max(mp, red);
    mq = team_max(mq, red);
    if (!isfinite(mp) || !isfinite(mq)) { finite = false; break; }
    if (mp * mq < P.tol) break;
  }

  // ---- F = (zS - H - tau g tau')^-1 and the parameter gradients
  gemm_la<OP_N, OP_N>(smem, n, n, n, g, n, taup, n, Y1, n);             // g tau'
  gemm_la<OP_N, OP_N>(smem, n, n, n, tau, n, Y1, n, W, n);              // tau g tau'
  for (int64_t e = team_tid(); e < n2; e += team_threads()) W[e] = csub(csub(cmul(z, S[e]), H[e]), W[e]);
  team_sync();
  bad |= cta_lu_inverse(W, F, n, smem_raw);
  gemm_la<OP_C, OP_N>(smem, n, n, n, F, n, lam, n, T1, n);              // F^H Lambda
  gemm_la<OP_N, OP_C>(smem, n, n, n, T1, n, F, n, gW, n, nullptr, 0, MONE);  // dW
  gemm_la<OP_N, OP_C>(smem, n, n, n, gW, n, Y1, n, T1, n, nullptr, 0, MONE);  // dtau = -dW (g tau')^H
  gemm_la<OP_N, OP_N>(smem, n, n, n, tau, n, g, n, Pm, n);              // tau g
  gemm_la<OP_C, OP_N>(smem, n, n, n, Pm, n, gW, n, Qm, n, nullptr, 0, MONE);  // dtau' = -(tau g)^H dW
  const cplx zc = cconj(z);
  for (int64_t e = team_tid(); e < n2; e += team_threads()) {
    const int64_t i = e / n, j = e % n;
    const cplx dw = gW[e], dt = T1[e], dtpH = cconj(Qm[j * n + i]);
    acc[0][e] = csub(acc[0][e], dw);                                      // H
    acc[2][e] = cadd(acc[2][e], cmul(zc, dw));                            // S
    acc[1][e] = csub(acc[1][e], cadd(dt, dtpH));                          // H01
    acc[3][e] = cadd(acc[3][e], cadd(cmul(zc, dt), cmul(z, dtpH)));       // S01
  }
  team_sync();
  if (team_tid() == 0) {
    P.status[idx] = bad ? NEGF_ERR_SINGULAR : (finite ? NEGF_OK : NEGF_ERR_NONFINITE);
    if (P.iters) P.iters[idx] = steps;
  }
}

__global__ void __launch_bounds__(CTA_THREADS, 1) lead_adjoint_kernel(const NegfLeadAdjProblem P) {
  char* const smem = negf_smem;
  __shared__ double red[CTA_THREADS / 32];
  cplx* slot = reinterpret_cast<cplx*>(P.scratch) + (size_t)(blockIdx.x / team_size()) * la_slot_elems(P);
  const size_t mn = (size_t)la_max_n(P.lead);
  for (size_t e = team_tid(); e < LA_NACC * mn * mn; e += team_threads()) slot[e] = cmk(0.0, 0.0);
  team_sync();
  for (int i = blockIdx.x / team_size(); i < P.n_items; i += gridDim.x / team_size()) la_item(P, i, slot, smem, red);
}

}  // namespace NEGF_NS
