// bound_kernel.cuh -- the score bound's kernel, instantiated in score_bound.cu (the default scores) and
// bound_forms.cu (the others).
#pragma once

#include "score_bound.cuh"

namespace sg {

const void* bound_form(const BoundJob& job);  // for scores other than the default ones; parameters (job, constants)

// One candidate per thread, blocks in list order (neighbouring candidates are of one read, or of
// reads of one length).
// C: the constants, BandBoundDefault for the default scores.
template <int H, bool WTD, class C>
__global__ void __launch_bounds__(128, H <= 4 ? 8 : H <= 8 ? 4 : 3)
    score_bound_kernel(BoundJob job, const __grid_constant__ BandConst bc) {
  const C c(bc);
  const int64_t n = job.n_dev ? *job.n_dev : job.n;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int r = job.read[t];
  const int L = job.lengths[r];
  int ub = 32767;
  const int lim = band_bound_limit(job.match, job.mismatch, L);
  if (lim > kBoundFloor - kBoundZero) {
    const int64_t win = max(job.diag[t] - job.I, -job.Is);  // run.c:667
    const int v = band_last_row<H, WTD>(job.gexp, win, job.rs + (int64_t)r * job.words,
                                        WTD ? job.ws + (int64_t)r * job.words : nullptr, L, c);
    if (v - kBoundZero < lim) ub = v - kBoundZero;
  }
  job.flag[t] = ub > job.min_score ? 1 : 0;
  job.ub[t] = (int16_t)ub;
}

template <class C>
inline const void* bound_kernel_of(const BoundJob& job) {
#define SG_BOUND(H) case H: return job.ws ? (const void*)score_bound_kernel<H, true, C> : (const void*)score_bound_kernel<H, false, C>;
  switch (job.H) {
    SG_BOUND(2)
    SG_BOUND(4)
    SG_BOUND(8)
    SG_BOUND(12)
  default: return nullptr;
  }
#undef SG_BOUND
}

}  // namespace sg
