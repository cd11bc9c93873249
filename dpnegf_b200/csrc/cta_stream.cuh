// CTA-wide elementwise passes streamed through shared memory.
//
// Plain per-thread global loads leave too few bytes in flight per SM (the
// form passes of the first kernel version were load-latency bound at
// ~25 GB/s per SM).  Here every thread stages its elements of 2048-element
// chunks with cp.async, two chunks in flight (128 KB per SM), and consumes
// exactly the elements it staged, so no barrier is needed inside the loop (a
// thread's own copies are complete behind its wait).
#pragma once
#include "negf_common.cuh"

namespace NEGF_NS {

constexpr int STREAM_CHUNK = 8 * TEAM_THREADS_PER_CTA;
constexpr int STREAM_SMEM_BYTES = 4 * STREAM_CHUNK * (int)sizeof(cplx);

// out[e] = alpha * (X[e] - z * Y[e]) for e < count; a null X or Y is zero.
// The chunks go round the team's CTAs.  Ends with team_sync().
// The roundings of z Y are spelled out, so that results do not depend on how the compiler contracts
// an instantiation: the products with Re z, the large ones, are fused into the sums.  The mixed sweep
// and the lead decimation amplify every rounding of their inputs and keep the imaginary part they
// have always had (MX).
template <bool MX = false>
NEGF_DEV void cta_shift_form(cplx* out, const cplx* X, const cplx* Y, cplx z, cplx alpha, int count,
                             cplx* smem) {
  const int tid = threadIdx.x;
  cplx* sx[2] = {smem, smem + STREAM_CHUNK};
  cplx* sy[2] = {smem + 2 * STREAM_CHUNK, smem + 3 * STREAM_CHUNK};
  const int all = (count + STREAM_CHUNK - 1) / STREAM_CHUNK;
  const int nch = (all - team_rank() + team_size() - 1) / team_size();  // this CTA's chunks
  auto issue = [&](int c) {
    const int base = (team_rank() + c * team_size()) * STREAM_CHUNK;
#pragma unroll
    for (int s = 0; s < STREAM_CHUNK / TEAM_THREADS_PER_CTA; ++s) {
      const int k = tid + s * TEAM_THREADS_PER_CTA, e = base + k;
      const bool v = e < count;
      if (X) cp_async16(sx[c & 1] + k, v ? X + e : X, v);
      if (Y) cp_async16(sy[c & 1] + k, v ? Y + e : Y, v);
    }
    cp_async_commit();
  };
  if (nch > 0) issue(0);
  for (int c = 0; c < nch; ++c) {
    if (c + 1 < nch) issue(c + 1);
    else cp_async_commit();
    cp_async_wait<1>();
    const int base = (team_rank() + c * team_size()) * STREAM_CHUNK;
#pragma unroll
    for (int s = 0; s < STREAM_CHUNK / TEAM_THREADS_PER_CTA; ++s) {
      const int k = tid + s * TEAM_THREADS_PER_CTA, e = base + k;
      if (e < count) {
        cplx x = X ? lds_after_wait(sx[c & 1] + k) : cmk(0.0, 0.0);
        cplx y = Y ? lds_after_wait(sy[c & 1] + k) : cmk(0.0, 0.0);
        const double re = __fma_rn(z.x, y.x, -__dmul_rn(z.y, y.y));
        const double im = MX ? __fma_rn(z.y, y.x, __dmul_rn(z.x, y.y)) : __fma_rn(z.x, y.y, __dmul_rn(z.y, y.x));
        out[e] = cmul(alpha, csub(x, cmk(re, im)));
      }
    }
  }
  cp_async_wait<0>();
  team_sync();
}

}  // namespace NEGF_NS
