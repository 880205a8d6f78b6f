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
#include "bound_kernel.cuh"

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

void launch_score_bound(const BoundJob& job, const BandConst& c, cudaStream_t st) {
  if (job.n <= 0) return;
  const void* k = band_is_default_bound(c) ? bound_kernel_of<BandBoundDefault>(job) : bound_form(job);
  if (!k) return;
  void* args[] = {(void*)&job, (void*)&c};
  cudaLaunchKernel(k, dim3((unsigned)((job.n + 127) / 128)), dim3(128), args, 0, st);  // errors surface at the caller's next check
}

}  // namespace sg
