// CTA-wide complex128 GEMM on FP64 tensor cores (DMMA m8n8k4), 3M products.
//
//   C[M x N] = alpha * op(A) * op(B) + beta * D        (D may alias C)
//
// One CTA of 256 threads (8 warps) walks the 64x64 output tiles of C; each
// tile streams 16-wide k-slabs of op(A) and op(B) into padded shared-memory
// tiles with cp.async (3-stage ring).  Each warp owns a 32x16 sub-tile and
// forms every complex product with three real DMMA m16n8k8 (Gauss/3M):
//   T1 = Ar*Br, T2 = Ai*Bi, T3 = (Ar+Ai)*(Br+Bi);  Re = T1-T2, Im = T3-T1-T2,
// or with four (4M) where an iteration amplifies the looser bound of 3M.  Other
// forms of the same code: CTAs of two warps with 32x32 tiles (NEGF_SMALL),
// clusters that deal the tiles round their CTAs (NEGF_TEAM), 32-row tiles of
// 16x16 sub-tiles (MI = 1) for few rows or even shares, and a drifting ring for
// ragged products (gemm_body).
// Shared-memory pitches are chosen so the DMMA fragment reads (one 16-byte
// complex per lane) are bank-conflict free for every operand orientation.
#pragma once
#include <type_traits>
#include "negf_common.cuh"

namespace NEGF_NS {

#ifndef NEGF_GT_K
#define NEGF_GT_K 16
#endif
constexpr int CTA_THREADS = TEAM_THREADS_PER_CTA;
#ifdef NEGF_SMALL
constexpr int GT_M = 32, GT_N = 32, GT_K = NEGF_GT_K;
#else
constexpr int GT_M = 64, GT_N = 64, GT_K = NEGF_GT_K;
#endif
static_assert(GT_K == 16 || GT_K == 32, "k slab of 16 or 32");
constexpr int PITCH_MK = GT_K + 4;  // [64 rows][GT_K k] tiles (pitch = 4 mod 8)
constexpr int PITCH_KN = GT_N + 2;  // [GT_K k][64 cols] tiles (pitch = 2 mod 8)
constexpr int GT_LOADS = GT_M * GT_K / CTA_THREADS;  // 16-byte copies per thread per operand tile
constexpr int GT_TILE = (GT_M * PITCH_MK > GT_K * PITCH_KN) ? GT_M * PITCH_MK : GT_K * PITCH_KN;
#ifndef NEGF_GT_STAGES
#define NEGF_GT_STAGES 3
#endif
// Depth of the cp.async k-slab ring; one value for the whole library (the host-side shared-memory
// sizes of every kernel derive from it).  4 stages measured 4 % slower on the 256^3 product and
// the sweep (LU solves 2 % faster).
constexpr int GT_STAGES = NEGF_GT_STAGES;
static_assert(GT_STAGES == 3 || GT_STAGES == 4, "3- or 4-stage ring");
constexpr int GEMM_SMEM_BYTES = 2 * GT_STAGES * GT_TILE * (int)sizeof(cplx);  // stages x (A,B)

struct GemmArgs {
  int M, N, K;
  const cplx* A;
  int64_t lda;
  const cplx* B;
  int64_t ldb;
  cplx* C;
  int64_t ldc;
  const cplx* D;  // addend, read only when use_d
  int64_t ldd;
  cplx alpha, beta;
  bool use_d;
};

NEGF_DEV GemmArgs gemm_args(int M, int N, int K, const cplx* A, int64_t lda, const cplx* B, int64_t ldb,
                            cplx* C, int64_t ldc) {
  GemmArgs g;
  g.M = M; g.N = N; g.K = K;
  g.A = A; g.lda = lda; g.B = B; g.ldb = ldb; g.C = C; g.ldc = ldc;
  g.D = nullptr; g.ldd = 0;
  g.alpha = cmk(1.0, 0.0); g.beta = cmk(0.0, 0.0); g.use_d = false;
  return g;
}

// op(A) tile element (m, k) -> shared-memory index
template <int OP>
NEGF_DEV int a_idx(int m, int k) { return OP == OP_C ? k * PITCH_KN + m : m * PITCH_MK + k; }
// op(B) tile element (k, n) -> shared-memory index
template <int OP>
NEGF_DEV int b_idx(int k, int n) { return OP == OP_C ? n * PITCH_MK + k : k * PITCH_KN + n; }

// Stage the (m0,k0) tile of op(A) into sA.
template <int OP, int TM = GT_M>
NEGF_DEV void load_a_tile(cplx* sA, const GemmArgs& g, int m0, int k0, int tid) {
#pragma unroll
  for (int s = 0; s < GT_LOADS * TM / GT_M; ++s) {
    int e = tid + s * CTA_THREADS;
    if (OP == OP_C) {  // stored X is K x M: tile rows k, cols m
      int r = e / TM, c = e % TM;
      int k = k0 + r, m = m0 + c;
      bool v = (k < g.K) && (m < g.M);
      const cplx* src = v ? g.A + (int64_t)k * g.lda + m : g.A;
      cp_async16(sA + r * PITCH_KN + c, src, v);
    } else {  // stored A is M x K: tile rows m, cols k
      int r = e / GT_K, c = e % GT_K;
      int m = m0 + r, k = k0 + c;
      bool v = (m < g.M) && (k < g.K);
      const cplx* src = v ? g.A + (int64_t)m * g.lda + k : g.A;
      cp_async16(sA + r * PITCH_MK + c, src, v);
    }
  }
}

// Stage the (k0,n0) tile of op(B) into sB.
template <int OP>
NEGF_DEV void load_b_tile(cplx* sB, const GemmArgs& g, int k0, int n0, int tid) {
#pragma unroll
  for (int s = 0; s < GT_LOADS; ++s) {
    int e = tid + s * CTA_THREADS;
    if (OP == OP_C) {  // stored X is N x K: tile rows n, cols k
      int r = e / GT_K, c = e % GT_K;
      int n = n0 + r, k = k0 + c;
      bool v = (n < g.N) && (k < g.K);
      const cplx* src = v ? g.B + (int64_t)n * g.ldb + k : g.B;
      cp_async16(sB + r * PITCH_MK + c, src, v);
    } else {  // stored B is K x N: tile rows k, cols n
      int r = e / GT_N, c = e % GT_N;
      int k = k0 + r, n = n0 + c;
      bool v = (k < g.K) && (n < g.N);
      const cplx* src = v ? g.B + (int64_t)k * g.ldb + n : g.B;
      cp_async16(sB + r * PITCH_KN + c, src, v);
    }
  }
}

struct Acc3M {
  double t1[2][2][4], t2[2][2][4], t3[2][2][4];  // [m16 frag][n8 frag][c0..c3]
  NEGF_DEV void zero() {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) t1[i][j][e] = t2[i][j][e] = t3[i][j][e] = 0.0;
  }
};

// Position in the warp's 32x16 sub-tile of accumulator element (i, j, e).
NEGF_DEV int acc_row(int i, int e, int wm, int lane) { return wm + 16 * i + (lane >> 2) + ((e & 2) ? 8 : 0); }
NEGF_DEV int acc_col(int j, int e, int wn, int lane) { return wn + 8 * j + 2 * (lane & 3) + (e & 1); }

// One warp's operand fragments for a k = 8 step of its 32x16 sub-tile (2 x 2 DMMA m16n8k8
// fragments per real plane), read through the index functors so the same code serves the GEMM
// tiles and the Gauss-Jordan panel update.
// G3 selects the complex product: Gauss/3M (three real MMAs, t1..t3) or the
// conventional 4M form (four real MMAs into t1 = Re, t2 = Im), whose
// componentwise error bound is tighter -- used where an iteration amplifies
// rounding (the lead decimation).
struct Frag8 {
  double ar[2][4], ai[2][4], as[2][4], br[2][2], bi[2][2], bs[2][2];  // as/bs: re + im (3M) or -im (4M, as)
};
template <bool CONJ_A, bool CONJ_B, bool G3, int MI = 2, class AIdx, class BIdx>
NEGF_DEV void frag8_load(Frag8& f, const cplx* sA, const cplx* sB, int ks, int wm, int wn, int lane, AIdx aidx,
                         BIdx bidx) {
  const int gr = lane >> 2, k0 = ks * 8 + (lane & 3);
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = wm + 16 * i + gr;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      cplx a = sA[aidx(r + ((e & 1) ? 8 : 0), k0 + ((e & 2) ? 4 : 0))];
      f.ar[i][e] = a.x;
      f.ai[i][e] = CONJ_A ? -a.y : a.y;
      f.as[i][e] = G3 ? f.ar[i][e] + f.ai[i][e] : -f.ai[i][e];
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int c = wn + 8 * j + gr;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      cplx b = sB[bidx(k0 + 4 * e, c)];
      f.br[j][e] = b.x;
      f.bi[j][e] = CONJ_B ? -b.y : b.y;
      if (G3) f.bs[j][e] = f.br[j][e] + f.bi[j][e];
    }
  }
}
template <bool G3, int MI = 2>
NEGF_DEV void frag8_mma(Acc3M& acc, const Frag8& f) {
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      dmma1688(acc.t1[i][j], f.ar[i], f.br[j]);
      if (G3) {
        dmma1688(acc.t2[i][j], f.ai[i], f.bi[j]);
        dmma1688(acc.t3[i][j], f.as[i], f.bs[j]);
      } else {
        dmma1688(acc.t1[i][j], f.as[i], f.bi[j]);
        dmma1688(acc.t2[i][j], f.ar[i], f.bi[j]);
        dmma1688(acc.t2[i][j], f.ai[i], f.br[j]);
      }
    }
}
template <bool CONJ_A, bool CONJ_B, bool G3 = true, class AIdx, class BIdx>
NEGF_DEV void warp_mma_3m(Acc3M& acc, const cplx* sA, const cplx* sB, int ksteps, int wm, int wn, int lane,
                          AIdx aidx, BIdx bidx) {
  for (int ks = 0; ks < ksteps; ++ks) {
    Frag8 f;
    frag8_load<CONJ_A, CONJ_B, G3>(f, sA, sB, ks, wm, wn, lane, aidx, bidx);
    frag8_mma<G3>(acc, f);
  }
}

// Complex value of accumulator element (i, j, e).
template <bool G3>
NEGF_DEV cplx acc_value(const Acc3M& acc, int i, int j, int e) {
  const double t1 = acc.t1[i][j][e], t2 = acc.t2[i][j][e];
  if (G3) return cmk(t1 - t2, acc.t3[i][j][e] - t1 - t2);
  return cmk(t1, t2);
}

// Visit every accumulator element of this warp: f(row, col, value).
template <bool G3, int MI = 2, class F>
NEGF_DEV void acc_foreach(const Acc3M& acc, int wm, int wn, int lane, F f) {
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) f(acc_row(i, e, wm, lane), acc_col(j, e, wn, lane), acc_value<G3>(acc, i, j, e));
}

struct AIdxOp0 { NEGF_DEV int operator()(int m, int k) const { return a_idx<OP_N>(m, k); } };
struct AIdxOpC { NEGF_DEV int operator()(int m, int k) const { return a_idx<OP_C>(m, k); } };
struct BIdxOp0 { NEGF_DEV int operator()(int k, int n) const { return b_idx<OP_N>(k, n); } };
struct BIdxOpC { NEGF_DEV int operator()(int k, int n) const { return b_idx<OP_C>(k, n); } };

// Default epilogue: C = alpha * acc + beta * D.
struct EpiStore {
  GemmArgs g;
  NEGF_DEV void operator()(int m, int n, cplx v) const {
    cplx o = cmul(g.alpha, v);
    if (g.use_d) o = cfma(g.beta, g.D[(int64_t)m * g.ldd + n], o);
    g.C[(int64_t)m * g.ldc + n] = o;
  }
};

// The same with the addend of a warp's sub-tile fetched before the first store, so that its reads are
// in flight together and not one behind another's store (same values).  For 4M products only: their
// two accumulator planes leave the registers for it; with three the main loop would lose more.
struct EpiAdd {
  typedef cplx Addend;
  GemmArgs g;
  NEGF_DEV cplx fetch(int m, int n) const { return g.D[(int64_t)m * g.ldd + n]; }
  NEGF_DEV void store(int m, int n, cplx v, cplx d) const {
    g.C[(int64_t)m * g.ldc + n] = cfma(g.beta, d, cmul(g.alpha, v));
  }
};
template <class Epi>
struct EpiTraits {
  template <class T> static char test(typename T::Addend*);
  template <class T> static long test(...);
  static constexpr bool two_phase = sizeof(test<Epi>(nullptr)) == 1;
};

// acc = op(A) op(B) over the whole M x N output by the whole CTA; epi(m, n, acc)
// is called once for every in-range element.  The output must not alias A or
// B.  Ends with __syncthreads(), so whatever epi wrote to global memory is
// visible to every thread of the CTA on return.  k-slabs flow through a
// GT_STAGES-deep cp.async ring with one barrier per slab.  Bound by the DMMA
// pipe; two forms with the same MMAs in the same order (bitwise equal results):
//
// DRIFT = false: the barrier stands at the head of the slab and every tile starts its own ring.
// DRIFT = true: the slabs of all output tiles form one sequence, so a tile's first slabs load while
// the tile before it finishes; the slab's barrier stands between the operand reads and the MMAs of
// its last k = 8 step, which cover its skew and the next slab's first reads; and a warp whose
// 32 x 16 sub-tile lies outside the product does no MMAs.  Warps w and w + 4 share a tensor core,
// so the second row of sub-tiles is rotated by two columns: the live warps of a ragged tile then
// spread over all four.
// Time of one n^3 product (148 CTAs with their own operands), DRIFT = false -> true: n = 16
// 3.3 -> 2.5 us, 32 5.4 -> 3.8, 96 53.9 -> 40.5, 115 75.1 -> 72.2, 128 74.1 -> 73.0, 256 545 -> 543
// (73 % of the DMMA peak); 4M products at 256 666 -> 644.  Inside the 3M sweep at n = 128 and 256,
// where registers are short, the drifting form is 2-4 % slower, so the sweep takes it for ragged
// products only (see gemm_ragged); the 4M lead kernels take it always (3.7 % at n = 256).
template <int OPA, int OPB, bool G3, bool DRIFT, int MI = 2, class Epi>
NEGF_DEV void gemm_body(const GemmArgs& g, const Epi& epi) {
  cplx* const smem = smem_cplx();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 16 * MI, wn = ((warp + (DRIFT ? 2 * (warp >> 2) : 0)) & 3) * 16;
  const int nk = (g.K + GT_K - 1) / GT_K;
  typedef typename std::conditional<OPA == OP_C, AIdxOpC, AIdxOp0>::type AI;
  typedef typename std::conditional<OPB == OP_C, BIdxOpC, BIdxOp0>::type BI;
  constexpr bool CA = (OPA != OP_N), CB = (OPB != OP_N);
  auto sA = [&](int s) { return smem + (2 * s) * GT_TILE; };
  auto sB = [&](int s) { return smem + (2 * s + 1) * GT_TILE; };

  if constexpr (!DRIFT) {
    for (int m0 = 0; m0 < g.M; m0 += GT_M) {
      for (int n0 = 0; n0 < g.N; n0 += GT_N) {
        __syncthreads();  // the previous tile's last slab is no longer being read
#pragma unroll
        for (int s = 0; s < GT_STAGES - 1; ++s) {
          if (s < nk) {
            load_a_tile<OPA>(sA(s), g, m0, s * GT_K, tid);
            load_b_tile<OPB>(sB(s), g, s * GT_K, n0, tid);
          }
          cp_async_commit();
        }
        Acc3M acc;
        acc.zero();
        for (int kt = 0; kt < nk; ++kt) {
          cp_async_wait<GT_STAGES - 2>();
          __syncthreads();
          const int nx = kt + GT_STAGES - 1;
          if (nx < nk) {
            load_a_tile<OPA>(sA(nx % GT_STAGES), g, m0, nx * GT_K, tid);
            load_b_tile<OPB>(sB(nx % GT_STAGES), g, nx * GT_K, n0, tid);
          }
          cp_async_commit();
          warp_mma_3m<CA, CB, G3>(acc, sA(kt % GT_STAGES), sB(kt % GT_STAGES), GT_K / 8, wm, wn, lane, AI(), BI());
        }
        acc_foreach<G3>(acc, wm, wn, lane, [&](int r, int c, cplx v) {
          int m = m0 + r, n = n0 + c;
          if (m < g.M && n < g.N) epi(m, n, v);
        });
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    return;
  }

#ifndef NEGF_TEAM
  if constexpr (G3) {  // nested tile loops: 2.5 % faster than the general form below in the sweep at n = 96
    // the next slab to load: its tile corner, k offset and ring stage
    int lm = 0, ln = 0, lk = 0, lst = 0;
    int left = ((g.M + GT_M - 1) / GT_M) * ((g.N + GT_N - 1) / GT_N) * nk;
    auto load_next = [&]() {
      if (left > 0) {
        load_a_tile<OPA>(sA(lst), g, lm, lk, tid);
        load_b_tile<OPB>(sB(lst), g, lk, ln, tid);
        --left;
        lst = lst + 1 == GT_STAGES ? 0 : lst + 1;
        lk += GT_K;
        if (lk >= g.K) {
          lk = 0;
          ln += GT_N;
          if (ln >= g.N) { ln = 0; lm += GT_M; }
        }
      }
      cp_async_commit();
    };
    __syncthreads();  // whatever used the ring's memory before is done with it
#pragma unroll
    for (int s = 0; s < GT_STAGES - 1; ++s) load_next();
    cp_async_wait<GT_STAGES - 2>();
    __syncthreads();
    int st = 0;
    for (int m0 = 0; m0 < g.M; m0 += GT_M) {
      for (int n0 = 0; n0 < g.N; n0 += GT_N) {
        if (m0 + wm >= g.M || n0 + wn >= g.N) {  // no output in this warp's sub-tile: keep the ring going
          for (int k0 = 0; k0 < g.K; k0 += GT_K) {
            load_next();
            cp_async_wait<GT_STAGES - 2>();
            __syncthreads();
            st = st + 1 == GT_STAGES ? 0 : st + 1;
          }
          continue;
        }
        Acc3M acc;
        acc.zero();
        for (int k0 = 0; k0 < g.K; k0 += GT_K) {
          const cplx *a = sA(st), *b = sB(st);
          warp_mma_3m<CA, CB, G3>(acc, a, b, GT_K / 8 - 1, wm, wn, lane, AI(), BI());
          load_next();
          Frag8 f;
          frag8_load<CA, CB, G3>(f, a, b, GT_K / 8 - 1, wm, wn, lane, AI(), BI());
          cp_async_wait<GT_STAGES - 2>();
          __syncthreads();
          frag8_mma<G3>(acc, f);
          st = st + 1 == GT_STAGES ? 0 : st + 1;
        }
        acc_foreach<G3>(acc, wm, wn, lane, [&](int r, int c, cplx v) {
          const int m = m0 + r, n = n0 + c;
          if (m < g.M && n < g.N) epi(m, n, v);
        });
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    return;
  }
#endif

  // Output tiles of TM rows, dealt round the team.  The next slab to load: its tile, k offset, stage.
  constexpr int TM = 32 * MI;
  const int tn = (g.N + GT_N - 1) / GT_N, tiles = ((g.M + TM - 1) / TM) * tn;
  int lt = team_rank(), lk = 0, lst = 0;
  auto load_next = [&]() {
    if (lt < tiles) {
      load_a_tile<OPA, TM>(sA(lst), g, (lt / tn) * TM, lk, tid);
      load_b_tile<OPB>(sB(lst), g, lk, (lt % tn) * GT_N, tid);
      lst = lst + 1 == GT_STAGES ? 0 : lst + 1;
      lk += GT_K;
      if (lk >= g.K) { lk = 0; lt += team_size(); }
    }
    cp_async_commit();
  };
  __syncthreads();  // whatever used the ring's memory before is done with it
  if (nk > 0) {
#pragma unroll
    for (int s = 0; s < GT_STAGES - 1; ++s) load_next();
  }
  cp_async_wait<GT_STAGES - 2>();
  __syncthreads();
  int st = 0;
  for (int t = team_rank(); t < tiles; t += team_size()) {
    const int m0 = (t / tn) * TM, n0 = (t % tn) * GT_N;
    if (m0 + wm >= g.M || n0 + wn >= g.N) {  // no output in this warp's sub-tile: keep the ring going
      for (int k0 = 0; k0 < g.K; k0 += GT_K) {
        load_next();
        cp_async_wait<GT_STAGES - 2>();
        __syncthreads();
        st = st + 1 == GT_STAGES ? 0 : st + 1;
      }
      continue;
    }
    Acc3M acc;
    acc.zero();
    for (int k0 = 0; k0 < g.K; k0 += GT_K) {
      const cplx *a = sA(st), *b = sB(st);
#pragma unroll
      for (int ks = 0; ks < GT_K / 8 - 1; ++ks) {
        Frag8 f;
        frag8_load<CA, CB, G3, MI>(f, a, b, ks, wm, wn, lane, AI(), BI());
        frag8_mma<G3, MI>(acc, f);
      }
      load_next();
      Frag8 f;
      frag8_load<CA, CB, G3, MI>(f, a, b, GT_K / 8 - 1, wm, wn, lane, AI(), BI());
      cp_async_wait<GT_STAGES - 2>();
      __syncthreads();
      frag8_mma<G3, MI>(acc, f);
      st = st + 1 == GT_STAGES ? 0 : st + 1;
    }
    if constexpr (EpiTraits<Epi>::two_phase) {
      cplx d[MI][2][4];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int m = m0 + acc_row(i, e, wm, lane), n = n0 + acc_col(j, e, wn, lane);
            d[i][j][e] = m < g.M && n < g.N ? epi.fetch(m, n) : cmk(0.0, 0.0);
          }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int m = m0 + acc_row(i, e, wm, lane), n = n0 + acc_col(j, e, wn, lane);
            if (m < g.M && n < g.N) epi.store(m, n, acc_value<G3>(acc, i, j, e), d[i][j][e]);
          }
    } else {
      acc_foreach<G3, MI>(acc, wm, wn, lane, [&](int r, int c, cplx v) {
        const int m = m0 + r, n = n0 + c;
        if (m < g.M && n < g.N) epi(m, n, v);
      });
    }
  }
  cp_async_wait<0>();
  team_sync();
}

// Whether the drifting form is the faster one for an M x N product of the sweep: the last row or
// column of tiles leaves at least half of its warps without output (remainder 1 .. 32 of 64).
NEGF_DEV bool gemm_ragged(int M, int N) { return ((M - 1) & (GT_M - 1)) < GT_M / 2 || ((N - 1) & (GT_N - 1)) < GT_N / 2; }

// The compiled products (arguments by reference: one copy per call instead of two).
template <int OPA, int OPB, bool G3, bool DRIFT, int MI, class Epi>
__device__ __noinline__ void cta_gemm_fn(const GemmArgs& gr, const Epi& er) {
  const GemmArgs g = gr;
  const Epi epi = er;
  gemm_body<OPA, OPB, G3, DRIFT, MI>(g, epi);
}
template <int OPA, int OPB, bool G3, bool DRIFT, int MI>
__device__ __noinline__ void cta_gemm_std(const GemmArgs& gr) {
  const GemmArgs g = gr;
  gemm_body<OPA, OPB, G3, DRIFT, MI>(g, EpiStore{g});
}

template <int OPA, int OPB, int MI>
__device__ __noinline__ void cta_gemm_add(const GemmArgs& gr) {  // 4M, with an addend
  const GemmArgs g = gr;
  gemm_body<OPA, OPB, false, true, MI>(g, EpiAdd{g});
}

#ifdef NEGF_TEAM
// Tiles of 32 rows instead of 64 where they even out what the team's CTAs get: the longest share,
// in units of 32-row tiles, is compared (a 64 x 64 product on two CTAs is one 32-row tile each).
NEGF_DEV bool team_half_tiles(int M, int N) {
  const int tn = (N + GT_N - 1) / GT_N, sz = team_size();
  const int full = (((M + 63) / 64) * tn + sz - 1) / sz, half = (((M + 31) / 32) * tn + sz - 1) / sz;
  return half < 2 * full;
}
#endif

// The product with a caller's epilogue.
template <int OPA, int OPB, bool G3, bool DRIFT, class Epi>
NEGF_DEV void cta_gemm_epi(const GemmArgs& g, const Epi& e) {
#ifdef NEGF_TEAM
  if (team_half_tiles(g.M, g.N)) cta_gemm_fn<OPA, OPB, G3, true, 1>(g, e);
  else cta_gemm_fn<OPA, OPB, G3, true, 2>(g, e);
#else
  cta_gemm_fn<OPA, OPB, G3, DRIFT, 2>(g, e);
#endif
}

// C = alpha op(A) op(B) + beta D (D may alias C; C must not alias A or B).
template <int OPA, int OPB, bool G3 = true>
NEGF_DEV void cta_gemm(const GemmArgs& g) {
#ifdef NEGF_TEAM
  const bool half = team_half_tiles(g.M, g.N);
#else
  // 4M products with few rows (the small updates of the lead LU): 16-row sub-tiles keep all eight
  // warps, or at 16 rows no idle halves of four, on the tensor cores
  const bool half = !G3 && g.M <= GT_M / 2;
#endif
  if constexpr (G3) {
#ifdef NEGF_TEAM
    if (half) cta_gemm_std<OPA, OPB, G3, true, 1>(g);
    else cta_gemm_std<OPA, OPB, G3, true, 2>(g);
#else
    if (gemm_ragged(g.M, g.N)) cta_gemm_std<OPA, OPB, G3, true, 2>(g);
    else cta_gemm_std<OPA, OPB, G3, false, 2>(g);
#endif
  } else if (g.use_d) {
    if (half) cta_gemm_add<OPA, OPB, 1>(g);
    else cta_gemm_add<OPA, OPB, 2>(g);
  } else {
    if (half) cta_gemm_std<OPA, OPB, G3, true, 1>(g);
    else cta_gemm_std<OPA, OPB, G3, true, 2>(g);
  }
}

}  // namespace NEGF_NS
