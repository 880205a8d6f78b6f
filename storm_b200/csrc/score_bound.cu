// score_bound.cu -- which passing candidates can score above -t: an upper bound of the full
// alignment's score, so that only the others are aligned with traceback.
//
// The replay drops every candidate whose score is not above the running threshold, which starts
// at -t and only rises (run.c:664-691): a candidate whose score is certainly at most -t changes
// nothing, whatever its bound and traceback are.  The score of a cell of the full alignment
// (alignment.c:488-632) is the cost of one path of pair scores and gaps; the bound is the best
// such path of the band with every restriction taken out that the packed form has no room for
// (the indel limit, the greedy choice of one direction per cell, the cost of turning from an
// insertion to a deletion, masked codes), so it is never below that score.
//   * Every quality level's pair scores come from one factor per read position (band_bound_consts:
//     the rounded products are at least the level's scores, equal at level 3).
//   * Values -248 .. 767 are exact.  Lower ones are raised to -248, which only raises the bound; a read
//     long enough to exceed 767 has a bound only below band_bound_limit.
// The bound also orders the work among the candidates kept: the replay's threshold rises to a
// read's fourth best score, and each round of the alignment takes only candidates whose bound is
// above the threshold the rounds before left (replay_kernel).
//
// Bound by the integer ALU pipe as the filter is, with the filter's recurrence: 3.5 ALU
// instructions per two cells where the full alignment needs about 28 and writes direction bits.
#include "score_bound.cuh"

namespace sg {

// one warp per read
__global__ void band_streams_kernel(ReadsDev rd, int H, int64_t words, uint32_t* __restrict__ rs,
                                    uint32_t* __restrict__ ws, BandConst c) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rd.n; r += nwarps) {
    const int L = rd.lengths[r];
    const uint8_t* cd = rd.codes + r * rd.cstride;
    const uint8_t* lv = ws && rd.levels ? rd.levels + r * rd.lstride : nullptr;
    auto nib = [&](int i) { return i < 0 || i >= L ? kBandPad : 4u + (uint32_t)code_at(cd, i); };
    auto fac = [&](int i) { return (uint32_t)c.wl[lv && i >= 0 && i < L ? code_at(lv, i) : 3]; };
    for (int64_t p = lane; p < words; p += 32) {
      const int i = (int)p;
      rs[r * words + p] = band_stream_word(nib(i - H - 1), nib(i - H), nib(i - 1), nib(i));
      if (ws) ws[r * words + p] = fac(i - H) | fac(i) << 16;
    }
  }
}

void launch_band_streams(const ReadsDev& rd, int H, int64_t words, uint32_t* rs, uint32_t* ws, const BandConst& c,
                         cudaStream_t st) {
  if (rd.n <= 0) return;
  const int64_t blocks = std::min<int64_t>((rd.n + 7) / 8, 148 * 32);
  band_streams_kernel<<<(unsigned)blocks, 256, 0, st>>>(rd, H, words, rs, ws, c);
}

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

void launch_score_bound(const BoundJob& job, const BandConst& c, cudaStream_t st) {
  if (job.n <= 0) return;
  const unsigned blocks = (unsigned)((job.n + 127) / 128);
#define SG_BOUND(H, C)                                                                  \
  case H:                                                                               \
    if (job.ws) score_bound_kernel<H, true, C><<<blocks, 128, 0, st>>>(job, c);         \
    else score_bound_kernel<H, false, C><<<blocks, 128, 0, st>>>(job, c);               \
    break;
#define SG_BOUNDS(C) \
  switch (job.H) {   \
    SG_BOUND(2, C)   \
    SG_BOUND(4, C)   \
    SG_BOUND(8, C)   \
    SG_BOUND(12, C)  \
  default: break;    \
  }
  if (band_is_default_bound(c)) { SG_BOUNDS(BandBoundDefault) } else { SG_BOUNDS(BandConst) }
#undef SG_BOUNDS
#undef SG_BOUND
}

}  // namespace sg
