// Shared device primitives for the NEGF kernels (sm_100a).
//
// Complex numbers are complex128 stored interleaved (re, im) as double2, the
// same layout torch.complex128 uses, so host tensors are passed through
// without conversion.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#define NEGF_DEV __device__ __forceinline__

// The CTA building blocks and the sweep compile twice: one CTA per work item (namespace negf), and,
// with NEGF_TEAM, a thread-block cluster per item (namespace negf_team), whose CTAs split the output
// tiles and the elementwise passes and repeat the small serial parts.  NEGF_SMALL compiles the sweep
// a third time, for blocks of up to 32: CTAs of two warps with 32 x 32 tiles, three to an SM.
#if defined(NEGF_TEAM)
#define NEGF_NS negf_team
#elif defined(NEGF_SMALL)
#define NEGF_NS negf_small
#else
#define NEGF_NS negf
#endif

namespace NEGF_NS {

#ifdef NEGF_SMALL
constexpr int TEAM_THREADS_PER_CTA = 64, MIN_CTAS = 3;
#else
constexpr int TEAM_THREADS_PER_CTA = 256, MIN_CTAS = 1;
#endif
#ifdef NEGF_TEAM
NEGF_DEV int team_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return (int)r;
}
NEGF_DEV int team_size() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
  return (int)r;
}
// Barrier over every thread of the team; global writes before it are visible to the team after it.
NEGF_DEV void team_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// The 8 bytes at `p` (this CTA's shared memory) as CTA `rank` of the team has them.
NEGF_DEV unsigned long long team_peek(const unsigned long long* p, int rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  unsigned long long v;
  asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.u64 %0, [r];\n\t}\n"
               : "=l"(v)
               : "r"(a), "r"(rank)
               : "memory");
  return v;
}
#else
NEGF_DEV constexpr int team_rank() { return 0; }
NEGF_DEV constexpr int team_size() { return 1; }
NEGF_DEV void team_sync() { __syncthreads(); }
#endif
NEGF_DEV int team_tid() { return team_rank() * TEAM_THREADS_PER_CTA + (int)threadIdx.x; }
NEGF_DEV int team_threads() { return team_size() * TEAM_THREADS_PER_CTA; }
NEGF_DEV int team_warp() { return team_tid() >> 5; }
NEGF_DEV int team_warps() { return team_threads() >> 5; }

typedef double2 cplx;

NEGF_DEV cplx cmk(double r, double i) { return make_double2(r, i); }
NEGF_DEV cplx cadd(cplx a, cplx b) { return cmk(a.x + b.x, a.y + b.y); }
NEGF_DEV cplx csub(cplx a, cplx b) { return cmk(a.x - b.x, a.y - b.y); }
NEGF_DEV cplx cmul(cplx a, cplx b) { return cmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
NEGF_DEV cplx cconj(cplx a) { return cmk(a.x, -a.y); }
NEGF_DEV cplx cneg(cplx a) { return cmk(-a.x, -a.y); }
NEGF_DEV cplx cscale(cplx a, double s) { return cmk(a.x * s, a.y * s); }
// a*b + c
NEGF_DEV cplx cfma(cplx a, cplx b, cplx c) {
  return cmk(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
// Reciprocal by Smith's scaling (avoids overflow in |a|^2).
NEGF_DEV cplx crcp(cplx a) {
  if (fabs(a.x) >= fabs(a.y)) {
    double r = a.y / a.x, den = a.x + a.y * r;
    return cmk(1.0 / den, -r / den);
  } else {
    double r = a.x / a.y, den = a.x * r + a.y;
    return cmk(r / den, -1.0 / den);
  }
}
NEGF_DEV double cabs1(cplx a) { return fabs(a.x) + fabs(a.y); }
NEGF_DEV bool cfinite(cplx a) { return isfinite(a.x) && isfinite(a.y); }

// The CTA's dynamic shared memory, shared by the CTA-wide building blocks one after another.
extern __shared__ __align__(1024) char negf_smem[];
NEGF_DEV cplx* smem_cplx() { return reinterpret_cast<cplx*>(negf_smem); }

// ---------------------------------------------------------------------------
// cp.async (16-byte, L2-only) with zero fill when the source is out of range.  The copy writes
// shared memory behind the compiler's back: the memory clobbers here and on the wait keep reads of
// the staged entries between them, also where a thread consumes its own copies without a barrier
// (which wait_group orders; without the clobbers some instantiations of the sweep had their reads
// moved ahead of the wait and returned wrong, varying blocks).
NEGF_DEV void cp_async16(void* smem_dst, const void* gmem_src, bool valid) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem_src), "r"(n) : "memory");
}
// Global load that the compiler may not sink below later volatile asm (the
// DMMAs): used to put a read-modify-write's reads in flight before the math.
NEGF_DEV cplx ldg_early(const cplx* p) {
  cplx v;
  asm volatile("ld.global.cg.v2.f64 {%0,%1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
// Shared-memory read of an entry that this thread staged itself, kept in program order with the wait
// and the next copies as they are (volatile).
NEGF_DEV cplx lds_after_wait(const cplx* p) {
  cplx v;
  asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];\n"
               : "=d"(v.x), "=d"(v.y)
               : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p)))
               : "memory");
  return v;
}
NEGF_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
NEGF_DEV void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------------------
// FP64 tensor-core MMA, D(8x8) += A(8x4, row) * B(4x8, col).
// Fragment ownership for lane l: A[l/4][l%4], B[l%4][l/4],
// C[l/4][2*(l%4) + {0,1}].
NEGF_DEV void dmma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// FP64 tensor-core MMA, D(16x8) += A(16x8, row) * B(8x8, col).
// Fragment ownership for lane l (g = l/4, t = l%4):
//   A: a0 (g, t), a1 (g+8, t), a2 (g, t+4), a3 (g+8, t+4)
//   B: b0 (t, g), b1 (t+4, g)
//   C: c0 (g, 2t), c1 (g, 2t+1), c2 (g+8, 2t), c3 (g+8, 2t+1)
NEGF_DEV void dmma1688(double* c, const double* a, const double* b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// Operand transforms for the tile GEMM.
enum Op : int { OP_N = 0, OP_C = 1 /* conjugate transpose */, OP_K = 2 /* conjugate */ };

// Per-CTA phase clocks (thread 0): the cycles since the previous mark are
// charged to the phase that just ended.  Every mark follows a __syncthreads.
enum Phase {
  PH_FORM = 0, PH_GEMM_FWD, PH_INV_STAGE, PH_INV_PANEL, PH_INV_UPDATE, PH_INV_GATHER,
  PH_GEMM_BWD, PH_LESSER, PH_DOS, PH_TRANS, PH_OTHER, PH_REFINE, NPH
};
struct PhaseClock {
  unsigned long long c[NPH];
  long long t0;
  bool on;
  NEGF_DEV void start(bool enable) {
    on = enable && threadIdx.x == 0;
    for (int i = 0; i < NPH; ++i) c[i] = 0;
    t0 = on ? clock64() : 0;
  }
  NEGF_DEV void mark(int ph) {
    if (on) {
      long long t = clock64();
      c[ph] += (unsigned long long)(t - t0);
      t0 = t;
    }
  }
};

// Reductions over the CTA (every thread gets the result; begin and end with a barrier).
NEGF_DEV double cta_max(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = red[0];
  for (int w = 1; w < TEAM_THREADS_PER_CTA / 32; ++w) s = fmax(s, red[w]);
  __syncthreads();
  return s;
}

NEGF_DEV double cta_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < TEAM_THREADS_PER_CTA / 32; ++w) s += red[w];
  __syncthreads();
  return s;
}

// The same over the team.
#ifdef NEGF_TEAM
static __shared__ unsigned long long team_slot;  // what the team's other CTAs may read of this one

// v of every CTA's thread 0, folded in rank order by every thread: each sees the same bits.
template <class F>
NEGF_DEV double team_fold(double v, F f) {
  if (threadIdx.x == 0) team_slot = (unsigned long long)__double_as_longlong(v);
  team_sync();
  double s = __longlong_as_double((long long)team_peek(&team_slot, 0));
  for (int r = 1; r < team_size(); ++r) s = f(s, __longlong_as_double((long long)team_peek(&team_slot, r)));
  team_sync();
  return s;
}
NEGF_DEV double team_max(double v, double* red) {
  return team_fold(cta_max(v, red), [](double x, double y) { return fmax(x, y); });
}
NEGF_DEV double team_sum(double v, double* red) {
  return team_fold(cta_sum(v, red), [](double x, double y) { return x + y; });
}
// rank 0's value of v (uniform in that CTA)
NEGF_DEV int team_from_first(int v) {
  if (threadIdx.x == 0) team_slot = (unsigned long long)(unsigned)v;
  team_sync();
  const int f = (int)(unsigned)team_peek(&team_slot, 0);
  team_sync();
  return f;
}
#else
NEGF_DEV double team_max(double v, double* red) { return cta_max(v, red); }
NEGF_DEV double team_sum(double v, double* red) { return cta_sum(v, red); }
#endif

}  // namespace NEGF_NS
