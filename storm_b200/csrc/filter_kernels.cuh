// filter_kernels.cuh -- the kernels of the banded filter, instantiated in sw_filter.cu (the default scores) and
// filter_forms.cu (the others), so that a process loads the code of the forms it runs.
#pragma once

#include <algorithm>

#include "map_kernels.cuh"
#include "sw_filter.cuh"
#include "filter_ref.cuh"
#include "filter_core.cuh"

namespace sg {

// the filter's kernel for a job that does not have the default scores or has a work cursor; parameters (job,
// sp), of which all but the scalar form take the first
const void* filter_form(const FilterJob& job, bool dpx);

// Candidates per thread: a block of 256 threads takes a tile of 256 * rows contiguous
// candidates (rows of 256: kFilterTile, or FilterJob.rows with a cursor).  Tiles go out in
// list order -- from a work cursor to a persistent grid (a block takes the next tile when all
// its warps are done with the last: uneven tiles balance), or by block index to a grid of one
// tile per block -- so the warps resident at any time work on neighbouring candidates: in a batch whose reads are grouped by length, an SM runs
// warps of one read length.  A grid-stride loop over a grid larger than the resident set makes
// every resident block walk the whole list instead, which mixes all lengths on every SM; on a
// 35-150 bp batch that ran the same instructions 1.48x slower, stalled on instruction fetch.
// The tile goes to the whole block, not warp by warp, for the same reason: the warps of a
// block start every tile together and stay close in the long unrolled band code (warps taking
// tiles one by one drift apart in it, which measured 5-15 % slower).
constexpr int kFilterTile = 8;  // rows of a tile unless FilterJob.rows says otherwise

// The block's tiles in list order: by block index, or with a cursor taken from it one at a
// time (all threads of the block make the same calls).  Taking the next tile ahead, to hide
// the atomic's round trip, measured no faster.
struct FilterTiles {
  unsigned long long* cursor;
  int64_t T;  // candidates per tile
  __device__ __forceinline__ int64_t first() { return cursor ? after() : (int64_t)blockIdx.x * T; }
  __device__ __forceinline__ int64_t after() {
    __shared__ unsigned long long s_tile;
    if (!cursor) return INT64_MAX;
    __syncthreads();  // every thread has read the previous tile
    if (threadIdx.x == 0) s_tile = atomicAdd(cursor, 1ull);
    __syncthreads();
    return (int64_t)s_tile * T;
  }
};

// one block's filter counters (cells, candidates, band cells) into the stats: three global
// atomics per block.  `counters` is uniform over the block.
__device__ __forceinline__ void add_filter_counters(unsigned long long* counters, unsigned long long cells,
                                                    unsigned long long cands, unsigned long long band) {
  __shared__ unsigned long long s[3];
  if (threadIdx.x == 0) { s[0] = 0; s[1] = 0; s[2] = 0; }
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) {
    cells += __shfl_xor_sync(0xffffffffu, cells, o);
    cands += __shfl_xor_sync(0xffffffffu, cands, o);
    band += __shfl_xor_sync(0xffffffffu, band, o);
  }
  if ((threadIdx.x & 31) == 0 && cands) {
    atomicAdd(&s[0], cells);
    atomicAdd(&s[1], cands);
    atomicAdd(&s[2], band);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s[1]) {
    atomicAdd(&counters[2], s[0]);
    atomicAdd(&counters[5], s[1]);
    atomicAdd(&counters[6], s[2]);
  }
}

// Calls body(t) for the block's candidates t < n: with a cursor (CURSOR) tiles of `rows` rows
// taken from it one after the other, else the one tile blockIdx.x of kFilterTile rows, or, where the
// list does not fill the GPU with such tiles, of as few rows as spread it over the grid (a thread takes
// its rows one after the other: 117,000 candidates of 300 colour reads 116 us with 8 rows, 34 with
// 2; beyond that size fewer rows than 8 ran the colour workload's filter 1 % slower).  One
// call site of body per instantiation (it is the long unrolled band code).  The one-tile form
// has no barrier; run through the cursor loop it measured 3 % slower.
constexpr int64_t kFilterShort = 148 * 3 * 256 * 8;
template <bool CURSOR, class Body>
__device__ __forceinline__ void for_filter_tiles(const FilterJob& job, int64_t n, int rows, Body body) {
  if constexpr (CURSOR) {
    FilterTiles tiles{job.cursor, 256 * (int64_t)rows};
    for (int64_t base = tiles.first(); base < n; base = tiles.after())
      for (int i = 0; i < rows; ++i) {
        const int64_t t = base + i * 256 + threadIdx.x;
        if (t >= n) break;
        body(t);
      }
  } else {
    const int64_t row = 256 * (int64_t)gridDim.x;  // candidates of one row of the grid
    const int mine = n > kFilterShort ? kFilterTile : (int)min((int64_t)kFilterTile, (n + row - 1) / row);
    const int64_t t0 = (int64_t)blockIdx.x * 256 * mine + threadIdx.x;
    for (int i = 0; i < mine; ++i) {
      const int64_t t = t0 + (int64_t)i * 256;
      if (t >= n) break;
      body(t);
    }
  }
}

// SHORT: the batch has reads shorter than W (band longer than the read), which take the
// stream-decoding variant; without them the kernel holds only the split-layout core and
// fits in 64 registers for W <= 8.  CURSOR: job.cursor is set (persistent grid).
template <int W, bool SHORT, bool CURSOR>
__global__ void __launch_bounds__(256, (W <= 8 ? 4 : 2)) filter_flat_dpx_kernel(FilterJob job) {
  const uint32_t T = (uint32_t)(job.fm & 0xff) | ((uint32_t)((256 - job.fx) & 0xff) << 8) |
                     ((uint32_t)((256 - job.fx) & 0xff) << 16) | ((uint32_t)((256 - job.fx) & 0xff) << 24);
  const uint32_t NFO = (uint32_t)(uint16_t)(-job.fo) * 0x10001u;
  uint32_t TLO, THI, NFE, CFO;  // NFE: -ext in both halves (both layouts)
  filter_split_consts(job.fm, job.fx, job.fo, job.fe, TLO, THI, NFE, CFO);
  unsigned long long cells = 0, cands = 0, band = 0;
  const int64_t n = job.n_dev ? (int64_t)*job.n_dev : job.n;
  for_filter_tiles<CURSOR>(job, n, job.rows > 0 ? job.rows : kFilterTile, [&](int64_t t) {
    const int r = job.fr[t];
    const int d = job.fd[t];
    const int L = job.lengths[r];
    const int64_t pos = (int64_t)d - job.Is;
    int mx;
    if (!SHORT || L >= W)
      mx = filter_split<W>(job.gexp, pos, job.rexp + (int64_t)r * job.rstride, L, TLO, THI, NFE, CFO);
    else
      mx = filter_dpx<W>(job.genome, pos, job.codes + (int64_t)r * job.cstride, job.cstride, L, T, NFE, NFO);
    job.flag[t] = mx > job.fthr ? 1 : 0;
    cells += (unsigned long long)(2 * W) * (unsigned long long)(L + W - 1);
    band += (unsigned long long)L * (2 * job.Is + 1);
    cands++;
  });
  if (job.counters) add_filter_counters(job.counters, cells, cands, band);
}

// The same over band_core.cuh's core: a candidate passes when a cell of the last row is infinite.
// C: the constants, BandFilterDefault for the default scores.  Three blocks per SM for W = 8 (72
// registers) and two for 16 measured best: 24.6 -> 24.0 ms and 102.4 -> 99.6 ms against four and
// three (colour workload's candidates, mixed ones).
template <int H, bool CURSOR, class C>
__global__ void __launch_bounds__(256, (H <= 2 ? 4 : H <= 4 ? 3 : 2)) filter_band_kernel(const __grid_constant__ FilterJob job) {
  constexpr int W = 2 * H;
  const C c(job.band);
  unsigned long long cells = 0, cands = 0, band = 0;
  const int64_t n = job.n_dev ? (int64_t)*job.n_dev : job.n;
  for_filter_tiles<CURSOR>(job, n, job.rows > 0 ? job.rows : kFilterTile, [&](int64_t t) {
    const int r = job.fr[t];
    const int64_t pos = (int64_t)job.fd[t] - job.Is;
    const int L = job.lengths[r];
    const int mx = band_last_row<H, false>(job.gexp, pos, job.bs + (int64_t)r * job.bwords, nullptr, L, c);
    job.flag[t] = mx >= kBandInf ? 1 : 0;
    cells += (unsigned long long)(2 * W) * (unsigned long long)(L + W - 1);
    band += (unsigned long long)L * (2 * job.Is + 1);
    cands++;
  });
  if (job.counters) add_filter_counters(job.counters, cells, cands, band);
}

// Plain 32-bit variant (any score values), the restatement in filter_ref.cuh.
template <bool CURSOR>
__global__ void filter_flat_scalar_kernel(FilterJob job, ScoreParams sp) {
  unsigned long long cells = 0, cands = 0, band = 0;
  const int64_t n = job.n_dev ? (int64_t)*job.n_dev : job.n;
  for_filter_tiles<CURSOR>(job, n, job.rows > 0 ? job.rows : kFilterTile, [&](int64_t t) {
    const int r = job.fr[t];
    const int L = job.lengths[r];
    job.flag[t] = sw_filter_dispatch_ext(job.W, job.genome, (int64_t)job.fd[t] - job.Is,
                                         job.codes + (int64_t)r * job.cstride, L, sp) ? 1 : 0;
    cells += (unsigned long long)(2 * job.W) * (unsigned long long)(L + job.W - 1);
    band += (unsigned long long)L * (2 * job.Is + 1);
    cands++;
  });
  if (job.counters) add_filter_counters(job.counters, cells, cands, band);
}

}  // namespace sg
