// sw_filter.cu -- the banded SW filter on packed 16-bit pairs (DPX), one candidate diagonal
// per thread over a flat candidate list, and the order-preserving compaction of the
// candidates that pass.
//
// Semantics: those of alignment_avx2__align_{hexa,octa,quad,pair} (alignment_simd.c:2613-3404)
// for one hit of W cells, as restated in filter_ref.cuh (sw_filter_one).  Here the W cells of
// one anti-diagonal step live in W/2 registers, two signed 16-bit cells each (filter_core.cuh):
//   * the per-cell score is one prmt whose selector is the difference of a read byte and a
//     genome byte (no compare, no branch);
//   * I = max(P, P of the neighbour cell, 0) with P = max(I[l-1] - ext, M[l-1] - open), and
//     M = max(M[l-2] + score, I) in one __viaddmax_s16x2; cells carry a bias of 256 so that the
//     gap subtractions are plain 32-bit adds;
//   * in the split layout used for reads of at least W codes (cells j and j + W/2 share a
//     register) the neighbour cell is in the neighbouring register, and the code streams move
//     by renaming registers; reads shorter than W use the adjacent-pair layout, which decodes
//     the packed 2-bit streams directly.
// The upper u8 saturation of the reference (adds at 255) is not reproduced: the threshold is
// at most 254, so the first cell that would saturate already has a value above it and the
// hit passes in both; cells are masked before they propagate, so an unmasked run and a
// saturating one agree on pass/fail.  Values stay below 2^15 when L * match < 32000 (checked
// by the host, which otherwise uses the plain 32-bit kernel).
#include <algorithm>

#include "map_kernels.cuh"
#include "sw_filter.cuh"
#include "filter_ref.cuh"
#include "filter_core.cuh"

namespace sg {

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

__global__ void expand_genome_kernel(const uint8_t* __restrict__ codes, int64_t n_codes, uint8_t* __restrict__ gexp) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_codes; i += (int64_t)gridDim.x * blockDim.x)
    gexp[i] = (uint8_t)(code_at(codes, i) * 0x11);
}

void launch_expand_genome(const uint8_t* codes, int64_t n_codes, uint8_t* gexp, cudaStream_t st) {
  if (n_codes <= 0) return;
  int64_t blocks = (n_codes + 255) / 256;
  if (blocks > 148 * 64) blocks = 148 * 64;
  expand_genome_kernel<<<(unsigned)blocks, 256, 0, st>>>(codes, n_codes, gexp);
}

// one warp per read: bytes 0xC4 + c * 0x11 for the L codes, 0xC4 (code 0) after
__global__ void expand_reads_kernel(ReadsDev rd, uint8_t* __restrict__ rexp, int64_t rstride) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rd.n; r += nwarps) {
    const int L = rd.lengths[r];
    const uint8_t* c = rd.codes + r * rd.cstride;
    uint32_t* o = reinterpret_cast<uint32_t*>(rexp + r * rstride);
    for (int64_t w = lane; w < rstride / 4; w += 32) {
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = (int)(4 * w + k);
        const uint32_t b = i < L ? 0xC4u + 0x11u * (uint32_t)code_at(c, i) : 0xC4u;
        v |= b << (8 * k);
      }
      o[w] = v;
    }
  }
}

void launch_expand_reads(const ReadsDev& rd, uint8_t* rexp, int64_t rstride, cudaStream_t st) {
  if (rd.n <= 0) return;
  int64_t blocks = (rd.n + 7) / 8;
  if (blocks > 148 * 32) blocks = 148 * 32;
  expand_reads_kernel<<<(unsigned)blocks, 256, 0, st>>>(rd, rexp, rstride);
}

// Plain 32-bit variant (any score values), the restatement in map_kernels.cu.
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

bool filter_dpx_ok(const ScoreParams& sp, int max_len) {
  return sp.fm <= 127 && sp.fx <= 128 && (int64_t)max_len * sp.fm < 32000 && sp.fe <= 32000 && sp.fo <= 32000;
}

// job.n: the candidates, or with job.n_dev an upper bound of them.  One tile per block, or with
// job.cursor at most the resident grid.
void launch_filter_flat_job(const FilterJob& job, const ScoreParams& sp, bool dpx, cudaStream_t st) {
  if (job.n <= 0) return;
  const int64_t tile = 256 * (int64_t)(job.cursor && job.rows > 0 ? job.rows : kFilterTile);
  int64_t blocks = (job.n + tile - 1) / tile;
  // a short list over every SM, down to one row per block
  if (!job.cursor) blocks = std::max(blocks, std::min<int64_t>((job.n + 255) / 256, kFilterShort / (256 * kFilterTile)));
  auto grid = [&](const void* k) {
    return (unsigned)(job.cursor ? std::min<int64_t>(blocks, resident_grid_of(k, 256, 0)) : blocks);
  };
#define SG_FILTER(K, ...) K<<<grid(reinterpret_cast<const void*>(K)), 256, 0, st>>>(__VA_ARGS__)
#define SG_FILTER_W(S, C)                                                \
  switch (job.W) {                                                       \
  case 2: SG_FILTER((filter_flat_dpx_kernel<2, S, C>), job); break;      \
  case 4: SG_FILTER((filter_flat_dpx_kernel<4, S, C>), job); break;      \
  case 8: SG_FILTER((filter_flat_dpx_kernel<8, S, C>), job); break;      \
  default: SG_FILTER((filter_flat_dpx_kernel<16, S, C>), job); break;    \
  }
  const bool cur = job.cursor != nullptr, shrt = job.min_len < job.W;
#define SG_FILTER_B(CUR, C)                                           \
  switch (job.band_H) {                                               \
  case 2: SG_FILTER((filter_band_kernel<2, CUR, C>), job); break;     \
  case 4: SG_FILTER((filter_band_kernel<4, CUR, C>), job); break;     \
  default: SG_FILTER((filter_band_kernel<8, CUR, C>), job); break;    \
  }
  if (job.band_H) {
    if (band_is_default_filter(job.band)) {
      if (cur) { SG_FILTER_B(true, BandFilterDefault) } else { SG_FILTER_B(false, BandFilterDefault) }
    } else {
      if (cur) { SG_FILTER_B(true, BandConst) } else { SG_FILTER_B(false, BandConst) }
    }
  } else if (!dpx) {
    if (cur) SG_FILTER(filter_flat_scalar_kernel<true>, job, sp);
    else SG_FILTER(filter_flat_scalar_kernel<false>, job, sp);
  } else if (!shrt) {
    if (cur) { SG_FILTER_W(false, true) } else { SG_FILTER_W(false, false) }
  } else {
    if (cur) { SG_FILTER_W(true, true) } else { SG_FILTER_W(true, false) }
  }
#undef SG_FILTER_B
#undef SG_FILTER_W
#undef SG_FILTER
}

// ------------------------------------------------------------------ compaction of passing candidates

// ------------------------------------------------------------------------------ selection
//
// The flagged candidates in order: a count per tile of 4,096 flag bytes, whose last block to finish scans
// the counts (it waits for nothing, the others are done) and applies the gates, then the writes.  The
// bytes are read twice where pass words, their scan (one to three launches), a gate and the writes took
// four to six launches: 10 us for 16 reads (269 candidates) against 14, 50 us for 12 million.  Launches
// count where a call is small: one of 16 reads went from 432 to 379 us with half of them gone.

constexpr int kSelectThreads = 256;
static_assert(kSelectTile == kSelectThreads * 16, "a thread takes 16 flag bytes");

// flags [t0, t0 + 16) of n as bits
__device__ __forceinline__ uint32_t flags16(const uint8_t* __restrict__ flag, int64_t t0, int64_t n) {
  uint32_t bits = 0;
  if (t0 + 16 <= n) {
    const uint4 q = *reinterpret_cast<const uint4*>(flag + t0);
    const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int b = 0; b < 4; ++b) bits |= ((v[k] >> (8 * b)) & 1u) << (4 * k + b);
  } else {
    for (int64_t t = t0; t < n; ++t) bits |= (uint32_t)(flag[t] & 1) << (t - t0);
  }
  return bits;
}

// exclusive scan over the block; *total the sum
template <class T>
__device__ __forceinline__ T select_scan(T v, T* wsum, T* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  __syncthreads();  // wsum is free again
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  T before = 0, all = 0;
#pragma unroll
  for (int k = 0; k < kSelectThreads / 32; ++k) {
    if (k < w) before += wsum[k];
    all += wsum[k];
  }
  *total = all;
  return before + incl - v;
}

__device__ __forceinline__ void apply_gate(const SelectGate& g, int64_t total) {
  if (!g.status) return;
  unsigned long long s = *g.status;
  if (total > g.cap) s |= 4;
  if (total > g.limit) s |= 2;
  *g.status = s;
  *g.take = s ? 0 : (unsigned long long)total;
  if (!s) *g.sum += (unsigned long long)total;
  if ((unsigned long long)total > *g.most) *g.most = (unsigned long long)total;
}

__global__ void __launch_bounds__(kSelectThreads) select_count_kernel(int64_t ncap, const unsigned long long* __restrict__ n_dev,
                                                                      const uint8_t* __restrict__ flag, int64_t* tile,
                                                                      unsigned long long* ticket, SelectGate g0, SelectGate g1) {
  __shared__ int64_t wsum[kSelectThreads / 32];
  __shared__ bool last;
  const int64_t n = n_dev ? min(ncap, (int64_t)*n_dev) : ncap;
  const int64_t nt = (n + kSelectTile - 1) / kSelectTile;
  for (int64_t t = blockIdx.x; t < nt; t += gridDim.x) {
    const int64_t mine = __popc(flags16(flag, t * kSelectTile + threadIdx.x * 16, n));
    int64_t all;
    select_scan<int64_t>(mine, wsum, &all);
    if (threadIdx.x == 0) tile[t] = all;
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1ull) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int64_t per = (nt + kSelectThreads - 1) / kSelectThreads;
  const int64_t a = min(nt, threadIdx.x * per), b = min(nt, a + per);
  int64_t sum = 0;
  for (int64_t t = a; t < b; ++t) sum += __ldcg(reinterpret_cast<const long long*>(tile + t));
  int64_t total;
  int64_t off = select_scan<int64_t>(sum, wsum, &total);
  for (int64_t t = a; t < b; ++t) {
    const int64_t c = __ldcg(reinterpret_cast<const long long*>(tile + t));
    tile[t] = off;
    off += c;
  }
  if (threadIdx.x == 0) {
    tile[(ncap + kSelectTile - 1) / kSelectTile] = total;
    apply_gate(g0, total);
    apply_gate(g1, total);
  }
}

__global__ void __launch_bounds__(kSelectThreads) select_write_kernel(
    int64_t ncap, const unsigned long long* __restrict__ n_dev, const uint8_t* __restrict__ flag,
    const int64_t* __restrict__ tile, const int32_t* __restrict__ fr, const int32_t* __restrict__ fd,
    int32_t* __restrict__ p_read, int32_t* __restrict__ p_diag, int64_t pcap, const int16_t* __restrict__ ub,
    int16_t* __restrict__ p_ub) {
  __shared__ int wsum[kSelectThreads / 32];
  const int64_t n = n_dev ? min(ncap, (int64_t)*n_dev) : ncap;
  const int64_t nt = (n + kSelectTile - 1) / kSelectTile, end = (ncap + kSelectTile - 1) / kSelectTile;
  for (int64_t t = blockIdx.x; t < nt; t += gridDim.x) {
    const int64_t base = tile[t], next = tile[t + 1 < nt ? t + 1 : end];
    if (next == base) continue;  // uniform over the block
    const int64_t t0 = t * kSelectTile + threadIdx.x * 16;
    uint32_t m = flags16(flag, t0, n);
    int all;
    int64_t o = base + select_scan<int>(__popc(m), wsum, &all);
    while (m && o < pcap) {
      const int64_t c = t0 + (__ffs(m) - 1);
      p_read[o] = fr[c];
      p_diag[o] = fd[c];
      if (p_ub) p_ub[o] = ub[c];
      ++o;
      m &= m - 1;
    }
  }
}

// The same by one block in one launch, tile after tile, for the lists of a call of few reads.
__global__ void __launch_bounds__(kSelectThreads) select_small_kernel(
    int64_t ncap, const unsigned long long* __restrict__ n_dev, const uint8_t* __restrict__ flag, SelectGate g0, SelectGate g1,
    const int32_t* __restrict__ fr, const int32_t* __restrict__ fd, int32_t* __restrict__ p_read,
    int32_t* __restrict__ p_diag, int64_t pcap, const int16_t* __restrict__ ub, int16_t* __restrict__ p_ub) {
  __shared__ int wsum[kSelectThreads / 32];
  const int64_t n = min(ncap, (int64_t)*n_dev);
  int64_t total = 0;
  for (int64_t base = 0; base < n; base += kSelectTile) {
    const int64_t t0 = base + threadIdx.x * 16;
    uint32_t m = flags16(flag, t0, n);
    int all;
    int64_t o = total + select_scan<int>(__popc(m), wsum, &all);
    total += all;
    while (m && o < pcap) {
      const int64_t c = t0 + (__ffs(m) - 1);
      p_read[o] = fr[c];
      p_diag[o] = fd[c];
      if (p_ub) p_ub[o] = ub[c];
      ++o;
      m &= m - 1;
    }
  }
  __syncthreads();  // every thread has its n
  if (threadIdx.x == 0) {
    apply_gate(g0, total);
    apply_gate(g1, total);
  }
}

void launch_select_small(int64_t ncap, const unsigned long long* n_dev, const uint8_t* flag, const SelectGate& g0,
                         const SelectGate& g1, const int32_t* fr, const int32_t* fd, int32_t* p_read, int32_t* p_diag,
                         int64_t pcap, const int16_t* ub, int16_t* p_ub, cudaStream_t st) {
  select_small_kernel<<<1, kSelectThreads, 0, st>>>(ncap, n_dev, flag, g0, g1, fr, fd, p_read, p_diag, pcap, ub, p_ub);
}

static unsigned select_grid(int64_t ncap) { return (unsigned)std::clamp<int64_t>(select_tiles(ncap), 1, 148 * 8); }

void launch_select_count(int64_t ncap, const unsigned long long* n_dev, const uint8_t* flag, int64_t* tile,
                         unsigned long long* ticket, const SelectGate& g0, const SelectGate& g1, cudaStream_t st) {
  select_count_kernel<<<select_grid(ncap), kSelectThreads, 0, st>>>(ncap, n_dev, flag, tile, ticket, g0, g1);
}

void launch_select_write(int64_t ncap, const unsigned long long* n_dev, const uint8_t* flag, const int64_t* tile,
                         const int32_t* fr, const int32_t* fd, int32_t* p_read, int32_t* p_diag, int64_t pcap,
                         const int16_t* ub, int16_t* p_ub, cudaStream_t st) {
  select_write_kernel<<<select_grid(ncap), kSelectThreads, 0, st>>>(ncap, n_dev, flag, tile, fr, fd, p_read, p_diag, pcap, ub,
                                                                    p_ub);
}

}  // namespace sg
