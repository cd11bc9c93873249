// CTA-wide complex128 matrix inverse: two-level blocked Gauss-Jordan with
// partial pivoting on FP64 tensor cores, and for FP64 blocks of up to 64 the same
// transform held in registers (cta_inverse_reg, described there).  The rest of this
// comment is about the first.
//
// The matrix W (n x n, row stride ldw) is a work buffer in global memory and
// is destroyed; the inverse is written to G.  Pivoting is implicit: rows never
// move in memory.  For logical column c the pivot is the unused physical row
// p(c) of largest |re|+|im| (LAPACK's izamax measure).  The sweep leaves the
// accumulated row transform T (T A = the pivot-row permutation of I) stored
// in place: column c of W holds column p(c) of T.  Since row i of A^-1 is row
// p(i) of T, the inverse is recovered by the gather
//     G[i][j] = W[p(i)][p^-1(j)],
// fused into the final store.
//
// Blocking.  Columns are taken in outer blocks of OB = 128 (the whole matrix
// when n <= 128).  Inside a block, panels of NB columns are factorised in
// shared memory and applied to the block's other columns only (rank-NB
// updates, k = NB).  The finished block transform is then applied to every
// column outside the block with one GEMM of depth k = OB at full tile-GEMM
// efficiency:
//     W[:, c] <- W[:, block] * W[block pivots, c] + (W[:, c] with the block's pivot rows zeroed),
// reading the block's pivot rows from a snapshot (they are overwritten by the
// same update).  Work: n^3 complex multiply-adds, as for an explicit inverse
// by LU.
//
// Panel factorisation in registers: every thread holds whole panel rows
// (row tid + 256 r, NB complex entries), so a column step is one broadcast of
// the scaled pivot row through shared memory and register-only updates; the
// pivot search for the next column uses the entries each thread just
// produced.  Two barriers per column.
#pragma once
#include "cta_gemm_tc.cuh"

namespace NEGF_NS {

#ifndef NEGF_INV_SMALL_NB
#define NEGF_INV_SMALL_NB 8
#endif
// Panel width of the Gauss-Jordan inverse for blocks of n <= 64 (the block inverse's leaves).
// Measured against 16-wide panels (every SM inverting its own matrices): 4-9 % faster for
// n = 32..64, 2-3 % for the block inverse of n = 128..192, equal at n = 256 and n = 16.
constexpr int INV_SMALL_NB = NEGF_INV_SMALL_NB;
static_assert(INV_SMALL_NB == 8 || INV_SMALL_NB == 16, "8- or 16-wide panels for small blocks");
constexpr int INV_OB = 128;      // default outer block (columns) of the two-level Gauss-Jordan
constexpr int INV_OB_MAX = 512;  // widest outer block (one block: no outer update for n <= 512)

// Shared memory: panel, R tiles, pivot row and multiplier columns, then the
// integer maps (piv, pinv, reductions).  The maps start above the outer
// update's GEMM staging area (the DMMA ring, or the tcgen05 planes with TC),
// which that GEMM overwrites while the update epilogue still reads pinv.
template <int NB>
struct InvLayout {
  static constexpr int PP = NB + 4;  // panel pitch (= 4 mod 8: conflict-free A fragments)
  static constexpr int RP = GT_N + 2;
  __host__ __device__ static int rows(int n) { return (n + GT_M - 1) / GT_M * GT_M; }
  __host__ __device__ static size_t panel_bytes(int n) {
    size_t b = (size_t)rows(n) * PP * sizeof(double2) + 2 * (size_t)NB * RP * sizeof(double2);
    return b + 2 * (size_t)rows(n) * sizeof(double2) + NB * sizeof(double2);  // multiplier columns, spare row
  }
  __host__ __device__ static size_t maps_offset(int n, bool tc) {
    const size_t b = panel_bytes(n), g = tc ? (size_t)TC_SMEM_BYTES : (size_t)GEMM_SMEM_BYTES;
    return b < g ? g : b;
  }
  __host__ __device__ static size_t bytes(int n, bool tc) {
    return maps_offset(n, tc) + (size_t)(2 * n + 64) * sizeof(int) + 16 * sizeof(double);
  }
};

// Largest footprint over every block size up to max_n: blocks of 65..256 use
// 32-wide panels, the others 16-wide panels, and a device may mix both.
inline size_t inv_smem_bytes_host(int max_n, bool tc = false) {
  size_t a = InvLayout<32>::bytes(max_n < 256 ? max_n : 256, tc);
  const size_t s = InvLayout<INV_SMALL_NB>::bytes(max_n < 64 ? max_n : 64, tc);
  if (s > a) a = s;
  if (max_n > 256) {
    const size_t b = InvLayout<16>::bytes(max_n, tc);
    if (b > a) a = b;
  }
  size_t g = tc ? (size_t)TC_SMEM_BYTES : (size_t)GEMM_SMEM_BYTES;  // the outer update runs a CTA GEMM
  return a > g ? a : g;
}

// Complex elements of the pivot-row snapshot the inverse needs (INV_OB x n).
__host__ __device__ inline size_t inv_snapshot_elems(int n) { return (size_t)INV_OB * n; }

struct PanelIdx {
  int pitch;
  NEGF_DEV int operator()(int m, int k) const { return m * pitch + k; }
};
struct RIdx {
  NEGF_DEV int operator()(int k, int n) const { return k * (GT_N + 2) + n; }
};

// argmax over (value, index) pairs: larger value wins, ties go to the lower index
NEGF_DEV void argmax_merge(double& v, int& i, double ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
NEGF_DEV void warp_argmax(double& v, int& i) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    double ov = __shfl_xor_sync(0xffffffffu, v, off);
    int oi = __shfl_xor_sync(0xffffffffu, i, off);
    argmax_merge(v, i, ov, oi);
  }
}
NEGF_DEV double pivot_measure(cplx a) {
  double v = cabs1(a);
  return (v == v) ? v : INFINITY;  // NaN pivots are taken (and flagged) first
}

// The same search on integer keys: a pivot measure is >= 0 or +inf, and for such doubles the
// order of the IEEE bit patterns read as signed 64-bit integers is the numeric order, so the
// winner (ties to the lower index) is the one the double comparison picks, while the compares
// and shuffles stay on the integer pipes instead of the long-latency FP64 ones.  -1 is "no
// candidate"; a key <= 0 (zero pivot) or >= PIVOT_KEY_INF (infinite or NaN) is singular.
constexpr long long PIVOT_KEY_INF = 0x7ff0000000000000LL;
NEGF_DEV long long pivot_key(cplx a) { return __double_as_longlong(pivot_measure(a)); }
NEGF_DEV void argmax_merge_key(long long& v, int& i, long long ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
NEGF_DEV void warp_argmax_key(long long& v, int& i) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const long long ov = __shfl_xor_sync(0xffffffffu, v, off);
    const int oi = __shfl_xor_sync(0xffffffffu, i, off);
    argmax_merge_key(v, i, ov, oi);
  }
}
NEGF_DEV bool pivot_key_singular(long long k) { return k <= 0 || k >= PIVOT_KEY_INF; }

// Outer-update epilogue: pivot rows of the block take the product, the other
// rows add it to their current value.
struct EpiGJ {
  cplx* W;
  int64_t ldw;
  const int* pinv;
  int c_lo, c_hi, col0;
  NEGF_DEV void operator()(int m, int n, cplx v) const {
    cplx* dst = W + (int64_t)m * ldw + col0 + n;
    const int lc = pinv[m];
    *dst = (lc >= c_lo && lc < c_hi) ? v : cadd(*dst, v);
  }
};

// Returns 0 on success, 1 if a zero or non-finite pivot was met.  Uniform
// across the CTA; ends with __syncthreads().  `snap` is global scratch of
// inv_snapshot_elems(n) complex elements (unused when n <= INV_OB).  TC runs
// the outer update on the tcgen05 3xTF32 GEMM (FP32-accurate products).
template <int NB, int RT, bool G3, bool TC>
__device__ __noinline__ int cta_inverse_nb(cplx* W, int64_t ldw, int n, cplx* G, int64_t ldg, char* smem_raw,
                                           PhaseClock* pc, cplx* snap, int ob_max) {
  constexpr int PP = InvLayout<NB>::PP;
  constexpr int RP = InvLayout<NB>::RP;
  constexpr int NWARP = CTA_THREADS / 32;
  static_assert(NB * RT <= 32, "a thread holds RT panel rows of NB complex entries (n <= 256 RT)");
  const int n_pad = InvLayout<NB>::rows(n);
  cplx* P = reinterpret_cast<cplx*>(smem_raw);
  cplx* Rb[2] = {P + (size_t)n_pad * PP, P + (size_t)n_pad * PP + NB * RP};
  cplx* qrow = Rb[1] + NB * RP;  // [NB] published pivot row of the current column
  int* piv = reinterpret_cast<int*>(smem_raw + InvLayout<NB>::maps_offset(n, TC));  // logical column -> physical row
  int* pinv = piv + n;                           // physical row -> logical column (-1: unused)
  int* red_i = pinv + n;                         // [2][NWARP] pivot candidates (double buffered)
  int* s_misc = red_i + 2 * NWARP;               // [1]: singular flag
  long long* red_v = reinterpret_cast<long long*>(s_misc + 48);  // [2][NWARP] pivot keys
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
  // Panel rows owned by this thread: tid + 256 r, r < RT (n <= 256 RT).
  // Bit r of `used` is set once that row has served as a pivot.
  unsigned used = 0u;
  int par = 0;

  for (int i = tid; i < n; i += CTA_THREADS) pinv[i] = -1;
  if (tid == 0) s_misc[1] = 0;
  __syncthreads();

  // Every thread merges the per-warp candidates (one barrier per pivot) and
  // marks the winner as used; thread 0 records it for the updates and gather.
  auto choose_pivot = [&](long long v, int i, int c) -> int {
    warp_argmax_key(v, i);
    if (lane == 0) { red_v[par * NWARP + warp] = v; red_i[par * NWARP + warp] = i; }
    __syncthreads();
    long long bv = red_v[par * NWARP];
    int bi = red_i[par * NWARP];
#pragma unroll
    for (int k = 1; k < NWARP; ++k) argmax_merge_key(bv, bi, red_v[par * NWARP + k], red_i[par * NWARP + k]);
    par ^= 1;
    if (tid == 0) {
      if (pivot_key_singular(bv)) s_misc[1] = 1;
      piv[c] = bi;
      pinv[bi] = c;
    }
    if (bi % CTA_THREADS == tid) used |= 1u << (bi / CTA_THREADS);
    return bi;
  };

  const int ob = n <= ob_max ? n : ob_max;
  for (int c_lo = 0; c_lo < n; c_lo += ob) {
    const int c_hi = min(c_lo + ob, n);
    for (int p0 = c_lo; p0 < c_hi; p0 += NB) {
      const int w = min(NB, c_hi - p0);
      // ---- stage the panel W[:, p0:p0+w) (zero padded to NB columns, n_pad rows)
      for (int e = tid; e < n_pad * NB; e += CTA_THREADS) {
        int i = e / NB, jj = e % NB;
        bool v = (jj < w && i < n);
        cp_async16(P + i * PP + jj, v ? W + (int64_t)i * ldw + p0 + jj : W, v);
      }
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
      // each thread takes its rows (tid + 256 r) of the panel into registers
      cplx row[RT][NB];
      cplx mm[RT];  // the rows' entries in the column being eliminated
      long long bv = -1;
      int bi = n;
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const int i = tid + CTA_THREADS * r;
#pragma unroll
        for (int k = 0; k < NB; ++k) row[r][k] = (i < n) ? P[i * PP + k] : cmk(0.0, 0.0);
        mm[r] = row[r][0];
        if (i < n && !((used >> r) & 1u)) argmax_merge_key(bv, bi, pivot_key(mm[r]), i);
      }
      int p = choose_pivot(bv, bi, p0);
      pc->mark(PH_INV_STAGE);

      // ---- unblocked Gauss-Jordan on the panel, in registers.  Column jj:
      // the pivot row's owner publishes q_k = P[p][k]/P[p][jj] (q_jj = 1/P[p][jj])
      // and keeps it as its row; every other row i does
      //     P[i][k] <- (k == jj ? 0 : P[i][k]) - m_i q_k,   m_i = P[i][jj],
      // and hands the next column's entry to the pivot search.
      for (int jj = 0; jj < w; ++jj) {
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          if (tid + CTA_THREADS * r == p) {
            const cplx d = crcp(mm[r]);
#pragma unroll
            for (int k = 0; k < NB; ++k) {
              const cplx q = (k == jj) ? d : cmul(row[r][k], d);
              row[r][k] = q;
              qrow[k] = q;
            }
          }
        }
        __syncthreads();
        const int nxt = jj + 1;
        bv = -1;
        bi = n;
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          const int i = tid + CTA_THREADS * r;
          cplx mnext = cmk(0.0, 0.0);
          if (i < n) {
            if (i != p) {
              const cplx m = mm[r];
#pragma unroll
              for (int k = 0; k < NB; ++k) {
                const cplx q = qrow[k];
                const cplx x = (k == jj) ? cmk(0.0, 0.0) : row[r][k];
                const cplx o = csub(x, cmul(m, q));
                row[r][k] = o;
                if (k == nxt) mnext = o;
              }
            } else {
#pragma unroll
              for (int k = 0; k < NB; ++k)
                if (k == nxt) mnext = row[r][k];
            }
            if (nxt < w && i != p && !((used >> r) & 1u)) argmax_merge_key(bv, bi, pivot_key(mnext), i);
          }
          mm[r] = mnext;
        }
        if (nxt < w) p = choose_pivot(bv, bi, p0 + nxt);
        else __syncthreads();  // qrow is rewritten by the next panel's first column
      }
      // the factorised panel goes back to shared memory as the update's A operand
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const int i = tid + CTA_THREADS * r;
        if (i < n_pad) {
#pragma unroll
          for (int k = 0; k < NB; ++k) P[i * PP + k] = row[r][k];
        }
      }
      __syncthreads();
      pc->mark(PH_INV_PANEL);

      // ---- apply the panel to the block's other columns, one 64-wide tile at a time
      auto load_r = [&](cplx* Rt, int c0) {
        for (int e = tid; e < NB * GT_N; e += CTA_THREADS) {
          int kk = e / GT_N, cc = e % GT_N;
          bool v = (kk < w && c0 + cc < c_hi);
          const cplx* src = v ? W + (int64_t)piv[p0 + kk] * ldw + c0 + cc : W;
          cp_async16(Rt + kk * RP + cc, src, v);
        }
        cp_async_commit();
      };
      int tiles[INV_OB_MAX / GT_N + 1];
      int ntile = 0;
      for (int c0 = c_lo; c0 < c_hi; c0 += GT_N) {
        const int c1 = min(c0 + GT_N, c_hi);
        if (!(c0 >= p0 && c1 <= p0 + w)) tiles[ntile++] = c0;
      }
      if (ntile > 0) load_r(Rb[0], tiles[0]);
      for (int t = 0; t < ntile; ++t) {
        const int c0 = tiles[t];
        cplx* Rt = Rb[t & 1];
        if (t + 1 < ntile) load_r(Rb[(t + 1) & 1], tiles[t + 1]);
        else cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        for (int r0 = 0; r0 < n; r0 += GT_M) {
          // fetch this warp's slice of W (the addend) ahead of the tensor-core work
          cplx old[2][2][4];
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                int row = r0 + acc_row(i, e, wm, lane), col = c0 + acc_col(j, e, wn, lane);
                old[i][j][e] = cmk(0.0, 0.0);
                if (row < n && col < c_hi) old[i][j][e] = ldg_early(W + (int64_t)row * ldw + col);
              }
          Acc3M acc;
          acc.zero();
          warp_mma_3m<false, false, G3>(acc, P + (size_t)r0 * PP, Rt, NB / 8, wm, wn, lane, PanelIdx{PP}, RIdx());
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                int row = r0 + acc_row(i, e, wm, lane), col = c0 + acc_col(j, e, wn, lane);
                if (row < n && col < c_hi && (col < p0 || col >= p0 + w)) {
                  cplx v = acc_value<G3>(acc, i, j, e);
                  int lc = pinv[row];
                  bool is_piv = (lc >= p0 && lc < p0 + w);
                  W[(int64_t)row * ldw + col] = is_piv ? v : cadd(old[i][j][e], v);
                }
              }
        }
        __syncthreads();  // R[t & 1] is refilled two tiles later
      }
      cp_async_wait<0>();
      // ---- write the factorised panel back
      for (int e = tid; e < n * NB; e += CTA_THREADS) {
        int i = e / NB, jj = e % NB;
        if (jj < w) W[(int64_t)i * ldw + p0 + jj] = P[i * PP + jj];
      }
      __syncthreads();
      pc->mark(PH_INV_UPDATE);
    }

    // ---- apply the block transform to the columns outside the block (k = block width)
    if (ob < n) {
      const int kb = c_hi - c_lo;
#pragma unroll 4
      for (int e = tid; e < kb * n; e += CTA_THREADS) {
        int kk = e / n, c = e % n;
        snap[e] = W[(int64_t)piv[c_lo + kk] * ldw + c];
      }
      __syncthreads();
      if (c_lo > 0) {
        GemmArgs g = gemm_args(n, c_lo, kb, W + c_lo, ldw, snap, n, W, ldw);
        if constexpr (TC) cta_gemm_tc_epi<OP_N, OP_N>(g, smem_raw, EpiGJ{W, ldw, pinv, c_lo, c_hi, 0});
        else cta_gemm_epi<OP_N, OP_N, G3, false>(g, EpiGJ{W, ldw, pinv, c_lo, c_hi, 0});
      }
      if (c_hi < n) {
        GemmArgs g = gemm_args(n, n - c_hi, kb, W + c_lo, ldw, snap + c_hi, n, W + c_hi, ldw);
        if constexpr (TC) cta_gemm_tc_epi<OP_N, OP_N>(g, smem_raw, EpiGJ{W, ldw, pinv, c_lo, c_hi, c_hi});
        else cta_gemm_epi<OP_N, OP_N, G3, false>(g, EpiGJ{W, ldw, pinv, c_lo, c_hi, c_hi});
      }
      pc->mark(PH_INV_UPDATE);
    }
  }

  // ---- undo the implicit pivoting while storing: G[i][j] = W[p(i)][p^-1(j)]
#pragma unroll 4
  for (int e = tid; e < n * n; e += CTA_THREADS) {
    int i = e / n, j = e % n;
    G[(int64_t)i * ldg + j] = W[(int64_t)piv[i] * ldw + pinv[j]];
  }
  const int flag = s_misc[1];
  __syncthreads();
  pc->mark(PH_INV_GATHER);
  return flag;
}

static __shared__ int inv_lost;  // a panel of an in-register inverse of this item never came

NEGF_DEV void mbar_init(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
NEGF_DEV void mbar_inval(unsigned long long* b) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(b)) : "memory");
}
NEGF_DEV void mbar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(b)) : "memory");
}
// Bounded wait for the barrier's first phase; false when the limit (about two seconds) expired.
NEGF_DEV bool mbar_wait_once(unsigned long long* b) { return tc_bar_wait(smem_addr(b), 0u); }

// Reciprocal of a pivot with one division: conj(a) / |a|^2 on a scaled by the power of two of its
// larger component (exact, so no overflow or underflow of |a|^2).
NEGF_DEV cplx crcp_scaled(cplx a) {
  const int e = max(__double2hiint(a.x) & 0x7ff00000, __double2hiint(a.y) & 0x7ff00000);
  const double s = __hiloint2double(0x7fe00000 - min(max(e, 0x00100000), 0x7fd00000), 0);  // 2^-exponent
  const double x = a.x * s, y = a.y * s;
  const double r = s / fma(x, x, y * y);
  return cmk(x * r, -y * r);
}

// f(integral_constant<int, 0>) ... f(integral_constant<int, N - 1>)
template <int N, class F>
NEGF_DEV void static_groups(F f) {
  if constexpr (N > 1) static_groups<N - 1>(f);
  f(std::integral_constant<int, N - 1>());
}

// Inverse of a block of n <= 64 held in registers, W -> G: blocked Gauss-Jordan with implicit
// partial pivoting (the in-place transform of the form above, PW columns to a panel).
//
// Lane l of warp w owns rows l + 32 a (a < RA) of columns CW w + j.  A warp holds whole columns, so
// it factorises its panels alone, with reductions and shuffles and no barrier, and publishes each
// with an mbarrier arrival; every other warp waits for panel t and applies it to its own columns,
//     x[i][j] = (i a pivot of the panel ? 0 : x[i][j]) + sum_s P[i][s] v_s,   v_s = x[p_s][j],
// where the pivot rows' entries are exchanged inside the warp.  Every panel has its own slot in
// shared memory, so the warps need not be in step.  The pivot is the row whose |re| + |im| has the
// largest leading 32 bits (within 2^-20 of the largest), the lowest lane among equals.  Returns 1
// after a singular pivot or an expired wait, which also sets inv_lost.
// Bound by the latency of the panel chain (per column a reduction, a reciprocal and a rank-1 step
// of PW columns).  Against the blocked form with 8-wide panels in shared memory, every SM inverting
// its own matrices: n = 16 22.7 -> 7.4 us, 32 47 -> 17, 64 108 -> 57; the block inverse built on it
// at n = 128 324 -> 219 us, at 256 1278 -> 1072.
template <int RA, int CW, int PW>
__device__ __noinline__ int cta_inverse_reg(const cplx* W, int64_t ldw, int n, cplx* G, int64_t ldg) {
  constexpr int NM = 32 * RA, NSUB = CW / PW, NW = CTA_THREADS / 32, NPAN = NW * NSUB;
  cplx* pan = smem_cplx();                      // [NPAN][PW][NM] factorised panels
  cplx* rows = pan + NPAN * PW * NM;                                  // [NW warps][PW][PW] pivot-row entries
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(rows + NW * PW * PW);  // [NPAN] panel published
  int* piv = reinterpret_cast<int*>(bar + NPAN);                      // [NW CW] logical column -> physical row
  int* pinv = piv + NW * CW;                                          // [NM] physical row -> logical column
  int* flag = pinv + NM;                                              // [0] singular pivot, [1] a panel never came
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cplx x[RA][CW];
#pragma unroll
  for (int a = 0; a < RA; ++a)
#pragma unroll
    for (int j = 0; j < CW; ++j) {
      const int i = lane + 32 * a, c = CW * warp + j;
      x[a][j] = (i < n && c < n) ? W[(int64_t)i * ldw + c] : cmk(0.0, 0.0);
    }
  unsigned used = 0u;  // bit a: row lane + 32 a has served as a pivot (or does not exist)
#pragma unroll
  for (int a = 0; a < RA; ++a)
    if (lane + 32 * a >= n) used |= 1u << a;
  __syncthreads();  // whatever used this shared memory before is done with it
  if (tid < NPAN) mbar_init(bar + tid, 1);
  if (tid < 2) flag[tid] = 0;
  __syncthreads();

  // Panel g of this warp (g a compile-time index, so that x stays in registers): factorise its
  // columns and publish them.
  auto factor = [&](auto g_c) {
    constexpr int g = decltype(g_c)::value;
    const int c0 = CW * warp + PW * g, w = min(PW, n - c0);
    if (w <= 0) return;
#pragma unroll
    for (int k = 0; k < PW; ++k) {
      if (k < w) {
        unsigned key[RA], best = 0u;
#pragma unroll
        for (int a = 0; a < RA; ++a) {
          key[a] = (used >> a) & 1u ? 0u : 1u + (unsigned)(pivot_key(x[a][g * PW + k]) >> 32);
          best = max(best, key[a]);
        }
        best = __reduce_max_sync(0xffffffffu, best);
        int p = 0;
#pragma unroll
        for (int a = RA - 1; a >= 0; --a) {
          const unsigned m = __ballot_sync(0xffffffffu, key[a] == best);
          if (m) p = 32 * a + __ffs(m) - 1;
        }
        cplx q[PW];
#pragma unroll
        for (int j = 0; j < PW; ++j) {
          q[j] = x[0][g * PW + j];
#pragma unroll
          for (int a = 1; a < RA; ++a)
            if (a == (p >> 5)) q[j] = x[a][g * PW + j];
          q[j].x = __shfl_sync(0xffffffffu, q[j].x, p & 31);
          q[j].y = __shfl_sync(0xffffffffu, q[j].y, p & 31);
        }
        const bool sing = pivot_key_singular(pivot_key(q[k]));
        const cplx d = crcp_scaled(q[k]);
#pragma unroll
        for (int j = 0; j < PW; ++j) q[j] = j == k ? d : cmul(q[j], d);
#pragma unroll
        for (int a = 0; a < RA; ++a) {
          const bool pr = lane + 32 * a == p;
          if (pr) used |= 1u << a;
          const cplx m = x[a][g * PW + k];
#pragma unroll
          for (int j = 0; j < PW; ++j) {
            const cplx y = j == k ? cmk(0.0, 0.0) : x[a][g * PW + j];
            const cplx o = cmk(fma(-m.x, q[j].x, fma(m.y, q[j].y, y.x)), fma(-m.x, q[j].y, fma(-m.y, q[j].x, y.y)));
            x[a][g * PW + j] = cmk(pr ? q[j].x : o.x, pr ? q[j].y : o.y);
          }
        }
        if (lane == 0) {
          piv[c0 + k] = p;
          pinv[p] = c0 + k;
          if (sing) flag[0] = 1;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < PW; ++k)
#pragma unroll
      for (int a = 0; a < RA; ++a) pan[(c0 + k) * NM + lane + 32 * a] = x[a][g * PW + k];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar + c0 / PW);
  };

  // Apply the published panel at column c0 to column group g of this warp.
  cplx* rv = rows + warp * PW * PW;
  auto apply = [&](auto g_c, int c0) {
    constexpr int g = decltype(g_c)::value;
    const int w = min(PW, n - c0);
    bool gone[RA];  // rows that are pivots of the panel
#pragma unroll
    for (int a = 0; a < RA; ++a) gone[a] = false;
#pragma unroll
    for (int s = 0; s < PW; ++s) {
      const int p = s < w ? piv[c0 + s] : -1;
#pragma unroll
      for (int a = 0; a < RA; ++a) {
        const bool is = lane + 32 * a == p;
        gone[a] |= is;
#pragma unroll
        for (int j = 0; j < PW; ++j)
          if (is) rv[s * PW + j] = x[a][g * PW + j];
      }
    }
    __syncwarp();
#pragma unroll
    for (int a = 0; a < RA; ++a) {
      if (gone[a]) used |= 1u << a;
#pragma unroll
      for (int j = 0; j < PW; ++j) {
        x[a][g * PW + j].x = gone[a] ? 0.0 : x[a][g * PW + j].x;
        x[a][g * PW + j].y = gone[a] ? 0.0 : x[a][g * PW + j].y;
      }
    }
#pragma unroll
    for (int s = 0; s < PW; ++s) {
      if (s < w) {
        cplx m[RA];
#pragma unroll
        for (int a = 0; a < RA; ++a) m[a] = pan[(c0 + s) * NM + lane + 32 * a];
#pragma unroll
        for (int j = 0; j < PW; ++j) {
          const cplx v = rv[s * PW + j];
#pragma unroll
          for (int a = 0; a < RA; ++a) x[a][g * PW + j] = cfma(m[a], v, x[a][g * PW + j]);
        }
      }
    }
    __syncwarp();  // rv is rewritten by the next call
  };

  constexpr std::integral_constant<int, 0> G0{};
  bool lost = false;
  // Panel g of warp w0: the owner factorises it (its first panel it has factorised already) and
  // applies it to its other column groups; the next panel's owner goes ahead after its first group.
  auto panel = [&](auto g_c, int w0) {
    constexpr int g = decltype(g_c)::value;
    const int c0 = CW * w0 + PW * g;
    if (c0 >= n || lost) return;
    if (warp == w0) {
      if constexpr (g > 0) factor(g_c);
      static_groups<NSUB>([&](auto h_c) {
        if constexpr (decltype(h_c)::value != g) apply(h_c, c0);
      });
    } else {
      const bool ok = mbar_wait_once(bar + c0 / PW);
      __syncwarp();
      lost = !__all_sync(0xffffffffu, ok);
      if (lost) return;
      apply(G0, c0);
      if (g == NSUB - 1 && warp == w0 + 1) factor(G0);
      static_groups<NSUB>([&](auto h_c) {
        if constexpr (decltype(h_c)::value != 0) apply(h_c, c0);
      });
    }
  };
  if (warp == 0) factor(G0);
  for (int w0 = 0; w0 < NW; ++w0) static_groups<NSUB>([&](auto g_c) { panel(g_c, w0); });
  if (lost) flag[1] = inv_lost = 1;
  __syncthreads();
  // G[i][j] = W[p(i)][p^-1(j)] (every CTA of a team holds the same result; one stores it)
  if (!flag[1] && team_rank() == 0) {
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        const int i = lane + 32 * a, c = CW * warp + j;
        if (i < n && c < n) G[(int64_t)pinv[i] * ldg + piv[c]] = x[a][j];
      }
  }
  const int f = flag[0] | flag[1];
  if (tid < NPAN) mbar_inval(bar + tid);
  team_sync();
  return f;
}

// G3: complex products of the rank updates (Gauss/3M or conventional 4M);
// TC: outer update on the tensor-core 3xTF32 GEMM.  ob: outer block width,
// a multiple of 32 up to INV_OB_MAX (narrower blocks move work from the
// panels' rank-NB updates to the outer GEMM; ob >= n leaves no outer update).
// With ob < n the snapshot needs ob x n complex elements.
template <bool G3 = true, bool TC = false>
NEGF_DEV int cta_inverse_pivoted(cplx* W, int64_t ldw, int n, cplx* G, int64_t ldg, char* smem_raw, PhaseClock* pc,
                                 cplx* snap, int ob) {
  // Narrow panels for small blocks (the mixed block inverse's 64-wide leaves): a column step's
  // latency chain is shorter (16-wide measured 22 % faster than 32-wide at n = 64, 8 % at
  // n = 128, where the rank-16 updates start to cost more; 8-wide another 4-9 % for n <= 64).
  // One register row per thread up to n = 256.
  if (n > 64 && n <= 256) return cta_inverse_nb<32, 1, G3, TC>(W, ldw, n, G, ldg, smem_raw, pc, snap, ob);
  if constexpr (TC) {
    if (n <= 64) return cta_inverse_nb<INV_SMALL_NB, 1, G3, TC>(W, ldw, n, G, ldg, smem_raw, pc, snap, ob);
  }
  return cta_inverse_nb<16, 2, G3, TC>(W, ldw, n, G, ldg, smem_raw, pc, snap, ob);
}
template <bool G3 = true, bool TC = false>
NEGF_DEV int cta_inverse(cplx* W, int64_t ldw, int n, cplx* G, int64_t ldg, char* smem_raw, PhaseClock* pc,
                         cplx* snap, int ob = INV_OB) {
  // Up to n = 64 the block fits the CTA's registers.  The mixed sweep keeps the panel form: its
  // FP32-accurate products amplify every rounding of the leaves, so its results would move.
  if constexpr (!TC) {
    if (n <= 64) {
#ifdef NEGF_SMALL
      const int f = n <= 8    ? cta_inverse_reg<1, 4, 4>(W, ldw, n, G, ldg)
                    : n <= 16 ? cta_inverse_reg<1, 8, 4>(W, ldw, n, G, ldg)
                              : cta_inverse_reg<1, 16, 4>(W, ldw, n, G, ldg);  // n <= 32
#else
      const int f = n <= 16   ? cta_inverse_reg<1, 2, 2>(W, ldw, n, G, ldg)
                    : n <= 32 ? cta_inverse_reg<1, 4, 4>(W, ldw, n, G, ldg)
                              : cta_inverse_reg<2, 8, 4>(W, ldw, n, G, ldg);
#endif
      pc->mark(PH_INV_PANEL);
      return f;
    }
  }
#if defined(NEGF_TEAM) || defined(NEGF_SMALL)
  return 1;  // not reached: a team's larger blocks go through the block inverse or one CTA's pivoted form
#else
  return cta_inverse_pivoted<G3, TC>(W, ldw, n, G, ldg, smem_raw, pc, snap, ob);
#endif
}

}  // namespace NEGF_NS
