// index_build.cu -- device-resident spaced-seed index of one reference sequence for one seed:
// a CSR table first[4^w + 1] (offsets) / map[] (positions, ascending per key), the layout of
// the reference's contiguous index (index.c:161-188, read by index__get_extern_next_hit,
// index.c:212-241).
//
// Build = seed keys of every indexed position (kernel) -> stable LSD radix sort of (key, pos)
// -> the runs of equal keys in the sorted list: their number and squared lengths (the repeat filter's
// exact integer moments; the host turns them into the largest admissible count), then the offsets.
// When the filter erases nothing the sorted positions are the map; else the kept ones are compacted.
// The key table is written once, from the sorted list (nothing else has its 4^w entries: for a
// 1 Mbp sequence and w = 12 the passes over them were most of the build).  HBM-streaming work; the
// seeds of a sequence share one wait for their moments.
#include <cmath>
#include <vector>

#include "index_build.cuh"
#include "radix.cuh"

namespace sg {

// Indexed positions come as intervals [a, b); t-th indexed position = a_k + (t - before_k).
// A warp takes consecutive t: the interval of its first is searched, the others walk on from it.
constexpr int kKeysPerLane = 8;
struct KeySeed {
  SeedRuns runs;
  int nruns;
  SeedDev seed;  // span above 32: code by code
};

__global__ void seed_keys_kernel(const uint8_t* __restrict__ codes, const int64_t* __restrict__ ia,
                                 const int64_t* __restrict__ ibefore, int nint, int64_t total,
                                 const __grid_constant__ KeySeed ks, uint32_t* __restrict__ keys,
                                 uint32_t* __restrict__ pos) {
  const int lane = threadIdx.x & 31;
  const int64_t tw = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * kKeysPerLane);
  if (tw >= total) return;
  int lo = 0, hi = nint - 1;
  while (lo < hi) {  // last interval with before <= the warp's first t
    const int mid = (lo + hi + 1) >> 1;
    if (ibefore[mid] <= tw) lo = mid; else hi = mid - 1;
  }
#pragma unroll
  for (int r = 0; r < kKeysPerLane; ++r) {
    const int64_t t = tw + 32 * r + lane;
    if (t >= total) return;
    while (lo + 1 < nint && ibefore[lo + 1] <= t) ++lo;
    const int64_t p = ia[lo] + (t - ibefore[lo]);
    uint32_t key = 0;
    if (ks.seed.span <= 32) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(codes) + (p >> 4);
      const uint32_t w0 = reverse_codes(__ldg(w)), w1 = reverse_codes(__ldg(w + 1)), w2 = reverse_codes(__ldg(w + 2));
      const int sh = 2 * (int)(p & 15);
      const uint64_t win = (uint64_t)__funnelshift_l(w1, w0, sh) << 32 | __funnelshift_l(w2, w1, sh);
      for (int c = 0; c < ks.nruns; ++c) key |= (uint32_t)(win >> ks.runs.r[c].x) & ks.runs.r[c].y;
    } else {
      for (int c = 0; c < ks.seed.n_care; ++c) key = (key << 2) | (uint32_t)code_at(codes, p + ks.seed.care[c]);
    }
    keys[t] = key;
    pos[t] = (uint32_t)p;
  }
}

// The key table is written in blocks of kKeyBlock keys; bound[b]: first index of the sorted list whose
// key is in block b or a later one.  A block with up to kKeyScan positions goes over them, 256 at a time;
// with more (a key of a long repeat: 4 million positions took 7 ms) it searches for each of its keys.
constexpr int kKeyBlock = 2048;
constexpr int64_t kKeyScan = 1 << 15;

// length of the run of equal keys that starts at t
__device__ __forceinline__ int64_t run_length(const uint32_t* __restrict__ skeys, int64_t n, int64_t t, uint32_t k) {
  int64_t d = 1;
  while (t + d < n && skeys[t + d] == k) d <<= 1;
  int64_t lo = d >> 1, hi = min(d, n - t);  // t + lo has the key (or lo = 0), t + hi has not
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (skeys[t + mid] == k) lo = mid; else hi = mid;
  }
  return hi;
}

constexpr int kStatsThreads = 256;

// out[0] += squared run lengths, out[1] += runs, out[2] = longest run; the blocks' bounds.
__global__ void run_stats_kernel(const uint32_t* __restrict__ skeys, int64_t n, int64_t nblocks,
                                 unsigned long long* __restrict__ out, int32_t* __restrict__ bound) {
  unsigned long long s2 = 0, runs = 0, longest = 0;
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
    const int64_t t = base + lane;
    const uint32_t k = t < n ? skeys[t] : 0u;
    uint32_t prev = __shfl_up_sync(0xffffffffu, k, 1);
    if (lane == 0 && t) prev = skeys[t - 1];
    const bool head = t < n && (t == 0 || prev != k);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    if (!head) continue;
    // up to the next head of the warp, else on from the warp's end
    const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;
    unsigned long long c;
    if (later) c = (unsigned long long)__ffs(later);
    else if (base + 32 >= n) c = (unsigned long long)(n - t);
    else c = skeys[base + 32] == k ? (unsigned long long)(32 - lane) + (unsigned long long)run_length(skeys, n, base + 32, k)
                                   : (unsigned long long)(32 - lane);
    s2 += c * c;
    runs++;
    longest = max(longest, c);
    for (int64_t b = t ? (int64_t)(prev / kKeyBlock) + 1 : 0; b <= (int64_t)(k / kKeyBlock); ++b) bound[b] = (int32_t)t;
    if (t + (int64_t)c == n)
      for (int64_t b = (int64_t)(k / kKeyBlock) + 1; b <= nblocks; ++b) bound[b] = (int32_t)n;
  }
  for (int o = 16; o > 0; o >>= 1) {
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    runs += __shfl_xor_sync(0xffffffffu, runs, o);
    longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  }
  // one update per block: by warp, the updates of three words by 19,000 warps took 36 us of the kernel's
  // 41 us at 1 Mbp
  __shared__ unsigned long long part[3][kStatsThreads / 32];
  const int w = threadIdx.x >> 5;
  if (lane == 0) { part[0][w] = s2; part[1][w] = runs; part[2][w] = longest; }
  __syncthreads();
  if (threadIdx.x < 3) {
    unsigned long long v = part[threadIdx.x][0];
    for (int k = 1; k < kStatsThreads / 32; ++k)
      v = threadIdx.x < 2 ? v + part[threadIdx.x][k] : max(v, part[threadIdx.x][k]);
    if (v && threadIdx.x < 2) atomicAdd(&out[threadIdx.x], v);
    if (v && threadIdx.x == 2) atomicMax(&out[2], v);
  }
}

// keys equal to k at t and before it
__device__ __forceinline__ int64_t run_length_back(const uint32_t* __restrict__ skeys, int64_t t, uint32_t k) {
  int64_t d = 1;
  while (t - d >= 0 && skeys[t - d] == k) d <<= 1;
  int64_t lo = d >> 1, hi = min(d, t + 1);  // t - lo has the key, t - hi has not
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (skeys[t - mid] == k) lo = mid; else hi = mid;
  }
  return hi;
}

// keep[t]: whether the key at t has at most cmax positions.  Every position looks for its run's ends by
// itself, unless the key cmax places on or back settles it: erased run by run, by the thread at its head, a
// key with 8 of 16 million positions took 120 ms.
__global__ void keep_runs_kernel(const uint32_t* __restrict__ skeys, int64_t n, int32_t cmax, uint8_t* __restrict__ keep) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = skeys[t];
    const bool more = (t + cmax < n && skeys[t + cmax] == k) || (t - cmax >= 0 && skeys[t - cmax] == k) ||
                      run_length(skeys, n, t, k) + run_length_back(skeys, t, k) - 1 > cmax;
    keep[t] = more ? 0 : 1;
  }
}

__global__ void kept_positions_kernel(const uint8_t* __restrict__ keep, const int32_t* __restrict__ off,
                                      const uint32_t* __restrict__ spos, int64_t n, int32_t* __restrict__ map) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n && keep[t]) map[off[t]] = (int32_t)spos[t];
}

// first[k] of a block of keys: the offset (off[t], or t without off) of the first position t whose key is
// k or a later one: the first positions of the keys present go to shared memory, and a suffix
// minimum gives the others theirs.  total: the offset after the last position.
__global__ void __launch_bounds__(256) key_table_kernel(const uint32_t* __restrict__ skeys, int64_t n, int64_t nkeys,
                                                        const int32_t* __restrict__ bound,
                                                        const int32_t* __restrict__ off, const int32_t* __restrict__ total,
                                                        int32_t* __restrict__ first) {
  constexpr int PER = kKeyBlock / 256;
  __shared__ int32_t at[kKeyBlock];
  __shared__ int32_t wmin[8];
  const int64_t k0 = (int64_t)blockIdx.x * kKeyBlock;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t lo = bound[blockIdx.x], hi = bound[blockIdx.x + 1];
  if (hi - lo <= kKeyScan) {
    for (int k = threadIdx.x; k < kKeyBlock; k += 256) at[k] = 0x7fffffff;
    __syncthreads();
    for (int64_t t = lo + threadIdx.x; t < hi; t += 256) {
      const uint32_t k = skeys[t];
      if (t == 0 || skeys[t - 1] != k) at[k - (uint32_t)k0] = (int32_t)t;
    }
  } else {
    // the first position in [lo, hi] whose key is this one or a later one, the thread's searches side by side
    int32_t a[PER], b[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) { a[i] = (int32_t)lo; b[i] = (int32_t)hi; }
    for (int64_t left = hi - lo; left > 0; left >>= 1) {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int32_t mid = (int32_t)(((int64_t)a[i] + b[i]) >> 1);
        const bool before = a[i] < b[i] && skeys[mid] < (uint32_t)(k0 + threadIdx.x + 256 * i);
        if (before) a[i] = mid + 1;
        else b[i] = min(b[i], mid);
      }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) at[threadIdx.x + 256 * i] = a[i];
  }
  __syncthreads();
  int32_t v[PER], m = 0x7fffffff;
#pragma unroll
  for (int i = PER - 1; i >= 0; --i) {  // thread-local suffix minima
    m = min(m, at[threadIdx.x * PER + i]);
    v[i] = m;
  }
  int32_t x = m;  // of the lanes from this one on
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_down_sync(0xffffffffu, x, o);
    if (lane + o < 32) x = min(x, y);
  }
  if (lane == 0) wmin[w] = x;
  int32_t after = __shfl_down_sync(0xffffffffu, x, 1);
  if (lane == 31) after = 0x7fffffff;
  __syncthreads();
  for (int q = w + 1; q < 8; ++q) after = min(after, wmin[q]);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int64_t t = min((int64_t)min(v[i], after), hi);
    at[threadIdx.x * PER + i] = !off ? (int32_t)t : t < n ? off[t] : *total;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kKeyBlock; k += 256)
    if (k0 + k <= nkeys) first[k0 + k] = at[k];
}

// Host simulation of the position loop of index.c:65-96 at interval granularity: windows are
// skipped while i + span >= start of the next masked region, i jumps to end-1 of that region
// (re-checking the following regions), and that position is indexed without re-testing the
// loop bound.  Returns the intervals of indexed positions, in increasing order.
void indexed_intervals(int64_t n_codes, int span, const int32_t* rs, const int32_t* re, int nreg,
                       std::vector<int64_t>& a, std::vector<int64_t>& b) {
  a.clear();
  b.clear();
  int64_t map_size = n_codes - span + 1;
  if (map_size <= 0 || span >= n_codes) return;
  int64_t i = 0;
  int r = 0;
  while (i < map_size) {
    int64_t trig = (r < nreg) ? std::max<int64_t>(i, (int64_t)rs[r] - span) : map_size;
    if (trig >= map_size) {
      a.push_back(i); b.push_back(map_size);
      break;
    }
    if (trig > i) { a.push_back(i); b.push_back(trig); }
    i = trig;
    while (r < nreg && i + span >= rs[r]) { i = (int64_t)re[r] - 1; r++; }
    if (!a.empty() && b.back() == i) b.back() = i + 1;
    else { a.push_back(i); b.push_back(i + 1); }
    i++;
  }
}

// Largest count c that the repeat filter keeps: c is erased iff c - avg > l * sd with
// avg = sum(c^2)/N^2 and sd^2 = sum_{c>0}(c - avg)^2 / N (index.c:117-155), both from the exact
// integer moments, compared in long double.
int32_t repeat_cutoff(int stdev_distance, int64_t N, unsigned long long s2, unsigned long long nocc) {
  if (stdev_distance <= 0 || N <= 0) return INT32_MAX;
  long double n = (long double)N;
  long double avg = (long double)s2 / n / n;
  long double var = ((long double)s2 - 2.0L * avg * n + (long double)nocc * avg * avg) / n;
  long double sd = sqrtl(var > 0 ? var : 0);
  auto erased = [&](long double c) { return (c - avg) > (long double)stdev_distance * sd; };
  long double guess = floorl(avg + (long double)stdev_distance * sd);
  if (guess > (long double)INT32_MAX) return INT32_MAX;
  if (guess < 0) guess = 0;
  int64_t c = (int64_t)guess;
  while (c + 1 <= INT32_MAX && !erased((long double)(c + 1))) c++;
  while (c > 0 && erased((long double)c)) c--;
  return (int32_t)c;
}

namespace {

// one seed's build between its sort and its fill; keys, bound and iv are in the build's one scratch block
struct Sorted {
  uint32_t *keys = nullptr, *pos = nullptr;
  int32_t* bound = nullptr;
  int64_t* iv = nullptr;
  int64_t total = 0, nblocks = 0;
};

unsigned blocks_of(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

// A seed's indexed positions: the intervals' starts, then the positions before each; their number.  With
// masked regions in ascending order it is at most the sequence's length; with regions out of order the
// walk jumps back and indexes positions again.
struct Positions {
  std::vector<int64_t> iv;
  int nint = 0;
  int64_t total = 0;
};

int sort_seed(const uint8_t* d_codes, const Positions& at, const SeedDev& seed, Sorted* so, unsigned long long* mom,
              uint32_t* scratch, int64_t room, cudaStream_t st, int64_t& L) {
  const int64_t total = at.total;
  so->total = total;
  so->nblocks = ((int64_t)1 << (2 * seed.weight)) / kKeyBlock + 1;  // the last one: the table's closing entry
  // The sorted list ends in its own arrays, whichever way the passes go; the other side of the sort is
  // scratch that every seed of the sequence uses.
  int64_t* const d_iv = so->iv;
  const int passes = (2 * seed.weight + kRadixBits - 1) / kRadixBits;
  uint32_t* const sk = scratch;
  uint32_t* const sv = sk + room;
  void* const tmp = sv + room;
  uint32_t *k0 = passes & 1 ? sk : so->keys, *v0 = passes & 1 ? sv : so->pos;
  uint32_t *k1 = passes & 1 ? so->keys : sk, *v1 = passes & 1 ? so->pos : sv;
  SG_CUDA(cudaMemcpyAsync(d_iv, at.iv.data(), sizeof(int64_t) * at.iv.size(), cudaMemcpyHostToDevice, st));
  KeySeed ks;
  ks.seed = seed;
  ks.nruns = seed.span <= 32 ? make_runs(seed, ks.runs) : 0;
  const int TB = 256;
  seed_keys_kernel<<<blocks_of(total, TB * kKeysPerLane), TB, 0, st>>>(d_codes, d_iv, d_iv + at.nint, at.nint, total, ks, k0, v0);
  radix_sort_pairs(k0, v0, k1, v1, total, 2 * seed.weight, tmp, st);
  run_stats_kernel<<<(unsigned)std::min<int64_t>(blocks_of(total, kStatsThreads), 148 * 16), kStatsThreads, 0, st>>>(so->keys, total,
                                                                                           so->nblocks, mom, so->bound);
  L += 2 + 3 * passes;
  SG_CUDA(cudaGetLastError());
  return 0;
}

// The map and the key table; where the repeat filter erases, `total` (on the device) gets the map's length.
// scratch, room: of the sorts, which are done.
int fill_seed(DevIndex* out, const Sorted& so, int32_t cmax, int64_t longest, int32_t* total, uint32_t* scratch, int64_t room,
              StreamScratch& S, int64_t& L) {
  cudaStream_t st = S.st;
  const int TB = 256;
  int32_t* off = nullptr;
  if (longest <= cmax) {  // nothing erased: the sorted positions are the map
    S.keep(so.pos);
    out->map = reinterpret_cast<int32_t*>(so.pos);
    out->n = so.total;
  } else {
    off = reinterpret_cast<int32_t*>(scratch);
    uint8_t* const keep = reinterpret_cast<uint8_t*>(scratch + room);
    int32_t* const tmp = reinterpret_cast<int32_t*>(scratch + 2 * room);  // the scan's: fewer words than the sort's
    SG_CUDA(cudaMallocAsync(&out->map, sizeof(int32_t) * so.total, st));
    keep_runs_kernel<<<(unsigned)std::min<int64_t>(blocks_of(so.total, TB), 148 * 16), TB, 0, st>>>(so.keys, so.total, cmax,
                                                                                                 keep);
    exclusive_scan<uint8_t, int32_t>(keep, off, so.total, total, tmp, st);
    kept_positions_kernel<<<blocks_of(so.total, TB), TB, 0, st>>>(keep, off, so.pos, so.total, out->map);
    L += 2 + scan_launches(so.total);
    S.give_back(so.pos);
  }
  key_table_kernel<<<(unsigned)so.nblocks, 256, 0, st>>>(so.keys, so.total, out->nkeys, so.bound, off, total, out->first);
  L++;
  SG_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace

int build_indexes(const uint8_t* d_codes, int64_t n_codes, const int32_t* rs, const int32_t* re, int nreg,
                  const SeedDev* seeds, int nseeds, int stdev_distance, DevIndex* out, cudaStream_t st,
                  int64_t* launches) {
  constexpr int kGroup = 4;  // seeds whose sorted lists are held at once (8 bytes per position each)
  std::vector<Positions> at(nseeds);
  int64_t room = 1, iv_words = 0;  // most indexed positions, interval words of a seed
  for (int q = 0; q < nseeds; ++q) {
    std::vector<int64_t> a, b;
    indexed_intervals(n_codes, seeds[q].span, rs, re, nreg, a, b);
    Positions& x = at[q];
    x.nint = (int)a.size();
    x.iv = a;
    for (size_t k = 0; k < a.size(); ++k) { x.iv.push_back(x.total); x.total += b[k] - a[k]; }
    if (x.total > INT32_MAX) { sg_set_error("sequence too long for 32-bit positions"); return STORMGPU_EINVAL; }
    room = std::max(room, x.total);
    iv_words = std::max(iv_words, (int64_t)x.iv.size());
  }
  // The tables and the lists that become maps come first, in one order, then one block for everything that a
  // build needs only while it runs: a rebuild then finds in the pool what the build before gave back.  With the
  // block first it was cut from the place of a table, and with a block for each the pool's order changed from
  // build to build; new memory was mapped (10 to 120 ms) now and then, or with tables of 1 GB and more each time.
  StreamScratch S(st);
  for (int q = 0; q < nseeds; ++q) {
    out[q].weight = seeds[q].weight;
    out[q].nkeys = (int64_t)1 << (2 * seeds[q].weight);
    SG_CUDA(cudaMallocAsync(&out[q].first, sizeof(int32_t) * (out[q].nkeys + 1), st));
  }
  std::vector<uint32_t*> pos(nseeds, nullptr);
  for (int q = 0; q < nseeds; ++q) {
    if (at[q].total > 0) SG_CUDA(S.alloc(&pos[q], at[q].total));
    else SG_CUDA(cudaMemsetAsync(out[q].first, 0, sizeof(int32_t) * (out[q].nkeys + 1), st));
  }
  const int held = std::min(kGroup, nseeds);
  int64_t most_keys = 0;
  for (int q = 0; q < nseeds; ++q) most_keys = std::max(most_keys, (int64_t)1 << (2 * seeds[q].weight));
  int64_t size = 0;
  auto take = [&](int64_t bytes) { const int64_t at = size; size += (bytes + 255) & ~255LL; return at; };
  const int64_t at_scratch = take(sizeof(uint32_t) * 2 * room + radix_tmp_bytes(room));
  const int64_t at_mom = take((sizeof(unsigned long long) * 3 + sizeof(int32_t)) * kGroup);
  const int64_t at_keys = take(0), key_bytes = ((int64_t)sizeof(uint32_t) * room + 255) & ~255LL;
  take(key_bytes * held);
  const int64_t at_bound = take(0), bound_bytes = ((int64_t)sizeof(int32_t) * (most_keys / kKeyBlock + 2) + 255) & ~255LL;
  take(bound_bytes * held);
  const int64_t at_iv = take(0), iv_bytes = ((int64_t)sizeof(int64_t) * iv_words + 255) & ~255LL;
  take(iv_bytes * held);
  uint8_t* block;
  SG_CUDA(S.alloc(&block, size));
  uint32_t* const scratch = reinterpret_cast<uint32_t*>(block + at_scratch);
  unsigned long long* const mom = reinterpret_cast<unsigned long long*>(block + at_mom);
  int32_t* const lengths = reinterpret_cast<int32_t*>(mom + 3 * kGroup);  // of the maps with erased keys
  int64_t L = 0;
  for (int s0 = 0; s0 < nseeds; s0 += kGroup) {
    const int ng = std::min(kGroup, nseeds - s0);
    Sorted so[kGroup];
    SG_CUDA(cudaMemsetAsync(mom, 0, sizeof(unsigned long long) * 3 * kGroup, st));
    for (int q = 0; q < ng; ++q) {
      so[q].keys = reinterpret_cast<uint32_t*>(block + at_keys + q * key_bytes);
      so[q].bound = reinterpret_cast<int32_t*>(block + at_bound + q * bound_bytes);
      so[q].iv = reinterpret_cast<int64_t*>(block + at_iv + q * iv_bytes);
      so[q].pos = pos[s0 + q];
      if (at[s0 + q].total == 0) continue;
      if (const int rc = sort_seed(d_codes, at[s0 + q], seeds[s0 + q], &so[q], mom + 3 * q, scratch, room, st, L)) return rc;
    }
    unsigned long long hm[3 * kGroup];
    SG_CUDA(cudaMemcpyAsync(hm, mom, sizeof(hm), cudaMemcpyDeviceToHost, st));
    SG_CUDA(cudaStreamSynchronize(st));
    bool erased = false;
    for (int q = 0; q < ng; ++q) {
      if (so[q].total == 0) continue;
      DevIndex* o = &out[s0 + q];
      o->positions_indexed = so[q].total;
      o->cmax = repeat_cutoff(stdev_distance, so[q].total, hm[3 * q], hm[3 * q + 1]);
      if (const int rc = fill_seed(o, so[q], o->cmax, (int64_t)hm[3 * q + 2], lengths + q, scratch, room, S, L)) return rc;
      erased |= (int64_t)hm[3 * q + 2] > o->cmax;
    }
    if (!erased) continue;
    int32_t hl[kGroup];
    SG_CUDA(cudaMemcpyAsync(hl, lengths, sizeof(hl), cudaMemcpyDeviceToHost, st));
    SG_CUDA(cudaStreamSynchronize(st));
    for (int q = 0; q < ng; ++q)
      if (so[q].total > 0 && (int64_t)hm[3 * q + 2] > out[s0 + q].cmax) out[s0 + q].n = hl[q];
  }
  if (launches) *launches += L;
  return 0;
}

}  // namespace sg
