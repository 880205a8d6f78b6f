// filter_forms.cu -- the filter's kernels for scores other than the default ones, with a work cursor, in the
// core of filter_core.cuh and on plain integers.
#include "filter_kernels.cuh"

namespace sg {

template <bool CURSOR, class C>
static const void* band_form(int H) {
  switch (H) {
  case 2: return (const void*)filter_band_kernel<2, CURSOR, C>;
  case 4: return (const void*)filter_band_kernel<4, CURSOR, C>;
  default: return (const void*)filter_band_kernel<8, CURSOR, C>;
  }
}

template <bool SHORT, bool CURSOR>
static const void* dpx_form(int W) {
  switch (W) {
  case 2: return (const void*)filter_flat_dpx_kernel<2, SHORT, CURSOR>;
  case 4: return (const void*)filter_flat_dpx_kernel<4, SHORT, CURSOR>;
  case 8: return (const void*)filter_flat_dpx_kernel<8, SHORT, CURSOR>;
  default: return (const void*)filter_flat_dpx_kernel<16, SHORT, CURSOR>;
  }
}

const void* filter_form(const FilterJob& job, bool dpx) {
  const bool cur = job.cursor != nullptr;
  if (job.band_H) {
    if (!cur) return band_form<false, BandConst>(job.band_H);
    return band_is_default_filter(job.band) ? band_form<true, BandFilterDefault>(job.band_H)
                                            : band_form<true, BandConst>(job.band_H);
  }
  if (!dpx) return cur ? (const void*)filter_flat_scalar_kernel<true> : (const void*)filter_flat_scalar_kernel<false>;
  if (job.min_len < job.W) return cur ? dpx_form<true, true>(job.W) : dpx_form<true, false>(job.W);
  return cur ? dpx_form<false, true>(job.W) : dpx_form<false, false>(job.W);
}

}  // namespace sg
