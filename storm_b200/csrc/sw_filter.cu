// sw_filter.cu -- the banded SW filter on packed 16-bit pairs (DPX), one candidate diagonal
// per thread over a flat candidate list, and the order-preserving compaction of the
// candidates that pass.
//
// Semantics: those of alignment_avx2__align_{hexa,octa,quad,pair} (alignment_simd.c:2613-3404)
// for one hit of W cells, as restated in filter_ref.cuh (sw_filter_one).  Bands of 4 cells and more with
// scores that have score bytes run on band_core.cuh, whose head describes its cells.  W = 2 and other scores
// run on filter_core.cuh, where the W cells of one anti-diagonal step live in W/2 registers, two signed
// 16-bit cells each:
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
#include "filter_kernels.cuh"

namespace sg {

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
  const void* k;
  if (job.band_H && !job.cursor && band_is_default_filter(job.band))
    k = job.band_H == 2   ? (const void*)filter_band_kernel<2, false, BandFilterDefault>
        : job.band_H == 4 ? (const void*)filter_band_kernel<4, false, BandFilterDefault>
                          : (const void*)filter_band_kernel<8, false, BandFilterDefault>;
  else
    k = filter_form(job, dpx);
  if (job.cursor) blocks = std::min<int64_t>(blocks, resident_grid_of(k, 256, 0));
  void* args[] = {(void*)&job, (void*)&sp};
  cudaLaunchKernel(k, dim3((unsigned)blocks), dim3(256), args, 0, st);  // errors surface at the caller's next check
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
