// gather.cu -- hit gather: for one read-strand, every (seed, read position) key's CSR list
// (index.c:212-241) shifted by the read position, merged into the ascending, de-duplicated
// diagonals that process_read's heap yields (run.c:577-698): a diagonal is kept iff it is
// strictly greater than the previous one in sorted order, the previous of the first being -I
// (run.c:617, :648, :697).
//
// One warp per read: keys computed from the packed read, CSR offsets read from the (L2-resident) key
// table, positions gathered straight into the warp's shared memory, reduced to the distinct
// diagonals there and appended to the flat candidate list, in no order: only a candidate that
// passes the filter needs its place among its read's (3 in 1,000 on the colour workload), and
// slot_lists_kernel gives it (map_kernels.cu).  Every lane looks up several (seed, position) keys
// before any result is used, so that a read costs two memory latencies (key table, positions) rather
// than two per seed.  Reads with more index positions than a warp can hold go to a
// block-per-read kernel (shared memory up to 4096 positions) and, beyond that, to slices in global
// memory; these append ascending diagonals.
#include <type_traits>

#include "gather.cuh"

namespace sg {


// Seed key at read position rp; codes beyond the read's end read as 0 (seed.c:203-213).
__device__ __forceinline__ uint32_t read_key(const SeedDev& s, const uint8_t* rd, int L, int rp) {
  uint32_t key = 0;
  for (int c = 0; c < s.n_care; ++c) {
    const int p = rp + s.care[c];
    key = (key << 2) | (uint32_t)(p < L ? code_at(rd, p) : 0);
  }
  return key;
}

// The same key from a register window: codes rp .. rp + 31 of a read staged in shared memory
// (4-byte aligned, readable for 12 bytes from word rp / 16), codes from L on masked to 0;
// one shift and mask per care position instead of a shared-memory load.  Seeds of span <= 32.
__device__ __forceinline__ uint32_t read_key_window(const SeedDev& s, const uint8_t* rd, int L, int rp) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(rd) + (rp >> 4);
  const uint64_t lo = (uint64_t)w[0] | ((uint64_t)w[1] << 32);
  const int sh = 2 * (rp & 15);
  uint64_t win = sh ? (lo >> sh) | ((uint64_t)w[2] << (64 - sh)) : lo;  // code rp + k at bits 2k
  const int lim = L - rp;
  if (lim < 32) win &= (1ull << (2 * lim)) - 1ull;
  uint32_t key = 0;
  for (int c = 0; c < s.n_care; ++c) key = (key << 2) | (uint32_t)((win >> (2 * s.care[c])) & 3u);
  return key;
}

__device__ __forceinline__ int seed_npos(const SeedDev& s, int L) {
  return s.n_positions ? s.n_positions : (L - s.span + 1 > 0 ? L - s.span + 1 : 0);
}

// (index offset, count, read position) of position t of seed s, with that seed's key table;
// `read` is staged in shared memory (see read_key_window)
__device__ __forceinline__ void item_lookup(const int32_t* __restrict__ first, const SeedDev& s, int t,
                                            const uint8_t* read, int L, int& a, int& cnt, int& rp) {
  a = 0; cnt = 0; rp = 0;
  if (t >= seed_npos(s, L)) return;
  rp = s.n_positions ? s.positions[t] : t;
  if (rp < 0 || rp >= L) return;
  const uint32_t key = s.span <= 32 ? read_key_window(s, read, L, rp) : read_key(s, read, L, rp);
  a = __ldg(first + key);
  cnt = __ldg(first + key + 1) - a;
}

// Place of U candidates of the warp's read in the flat list (-1: the list is full).
__device__ __forceinline__ int64_t reserve(const GatherOut& go, int U) {
  unsigned long long base = 0;
  if ((threadIdx.x & 31) == 0 && U) base = atomicAdd(&go.counters[7], (unsigned long long)U);
  base = __shfl_sync(0xffffffffu, base, 0);
  if ((int64_t)(base + U) > go.cap) {
    if ((threadIdx.x & 31) == 0) atomicExch(&go.counters[8], 1ull);
    return -1;
  }
  return (int64_t)base;
}

constexpr int32_t kEmptySlot = 0x7fffffff;  // no diagonal (position - read position) reaches it

// The distinct values of a[0..H) stay, the repeats become kEmptySlot (one warp).  Rounds of claims
// without atomics: every undecided entry writes its index to tab[hash], and reads back who wrote
// last: itself -- it stays; an entry of its own value -- it is a repeat; another value -- it is undecided
// and goes to the next round, with another hash.  Every slot read was written in the same round, so
// the table is never cleared; all entries of one value are decided in the same round.  About 85 %
// are decided in the first.  The diagonal a read truly maps to comes once per (seed, position) that
// hits it: with an open-addressing set those lanes queue on one shared atomic.  list[0..H): the
// undecided entries.  Returns the number of distinct values.
__device__ __forceinline__ int warp_distinct(int32_t* a, int H, uint16_t* tab, int size, uint16_t* list) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  int U = 0, n = H;
  uint32_t mul = 0x9E3779B1u;
  for (int round = 0; n > 0; ++round) {
    for (int k = lane; k < n; k += 32) {
      const int i = round ? list[k] : k;
      tab[__umulhi((uint32_t)a[i] * mul, (uint32_t)size)] = (uint16_t)i;
    }
    __syncwarp();
    int left = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
      const int k = k0 + lane;
      bool stays = false, undecided = false, repeat = false;
      int i = 0;
      if (k < n) {
        i = round ? list[k] : k;
        const int32_t v = a[i];
        const int win = tab[__umulhi((uint32_t)v * mul, (uint32_t)size)];
        const int32_t wv = a[win];
        stays = win == i;
        undecided = wv != v && wv != kEmptySlot;
        repeat = !stays && !undecided;
      }
      // repeats are blanked after the chunk's reads; a blanked winner cannot be: winners stay
      const unsigned mu = __ballot_sync(0xffffffffu, undecided);
      U += __popc(__ballot_sync(0xffffffffu, stays));
      if (repeat) a[i] = kEmptySlot;
      if (undecided) list[left + __popc(mu & lt)] = (uint16_t)i;  // writes trail the reads
      left += __popc(mu);
      __syncwarp();
    }
    n = left;
    mul = mul * 0x85EBCA6Bu + 2u;  // odd
  }
  return U;
}

// A seed's care positions as runs, for keys from a window of 32 codes whose first code is in the
// high bits: the key is the OR of (window >> shift) & mask over the runs (4 to 7 of them, where taking
// the care positions one by one takes 10 to 15 steps).
struct SeedRuns {
  uint2 r[16];  // shift, mask; unused ones have mask 0
};

// returns the number of runs
__device__ __forceinline__ int make_runs(const SeedDev& s, SeedRuns& o) {
  int n = 0;
  for (int c = 0; c < 16; ++c) o.r[c] = make_uint2(0, 0);
  for (int c = 0; c < s.n_care;) {
    int m = 1;
    while (c + m < s.n_care && s.care[c + m] - s.care[c] == m) ++m;
    o.r[n++] = make_uint2((uint32_t)(62 - 2 * (s.care[c] + s.n_care - 1 - c)),
                          (uint32_t)((1ull << (2 * m)) - 1ull) << (2 * (s.n_care - c - m)));
    c += m;
  }
  return n;
}

// 16 packed codes, first code in the low bits -> first code in the high bits
__device__ __forceinline__ uint32_t reverse_codes(uint32_t x) {
  x = __brev(x);
  return ((x & 0x55555555u) << 1) | ((x >> 1) & 0x55555555u);
}

constexpr int kGWarps = 4;
// Reads per steal (GatherOut.reads_per_steal, 4 by default): the grid is the resident set, and
// every warp takes the next reads_per_steal reads (in the order of rd.order, or of the batch) from a work cursor until none is left, so
// reads with many index positions balance out, and warps append their candidates in close to
// read order: a batch whose reads are grouped by length gives a candidate list grouped by
// length, which the filter needs to keep one read length per SM.
constexpr int kReadBytes = STORMGPU_MAX_READ_LEN / 4 + 16;
constexpr int kReadWords = STORMGPU_MAX_READ_LEN / 16 + 3;

constexpr int kItems = 4;  // (seed, position) items per lane and round: 128 key lookups in flight per warp
constexpr int kChunks = 4; // chunks of 32 index positions loaded before any is used

// Words of a warp's shared memory for `cap` index positions: the positions; the claims of
// warp_distinct (16 bits each), whose space holds the item markers before (a byte per position); two
// words per item of a round, whose space holds the undecided entries (16 bits each) after.
__host__ __device__ constexpr int gather_half_words(int cap) { return (cap / 2 + 32) & ~31; }
__host__ __device__ constexpr int gather_item_words(int cap) {
  return gather_half_words(cap) > 2 * 32 * kItems ? gather_half_words(cap) : 2 * 32 * kItems;
}
__host__ __device__ constexpr int gather_warp_words(int cap) {
  return ((cap + 31) & ~31) + gather_half_words(cap) + gather_item_words(cap);
}

__global__ void __launch_bounds__(kGWarps * 32, 9) gather_fused_kernel(ReadsDev rd, IndexView ix, int I, GatherOut go,
                                                                   const __grid_constant__ SeedSet gs) {
  extern __shared__ __align__(16) int32_t sm[];  // gather_warp_words per warp
  __shared__ SeedRuns runs[kMaxSeeds];
  __shared__ int32_t sspan[kMaxSeeds];
  __shared__ int s_nruns;
  __shared__ int32_t soff[kGWarps][kMaxSeeds + 1];  // first item of every seed, for the current read
  __shared__ const int32_t* s_first[kMaxSeeds];
  __shared__ const int32_t* s_map[kMaxSeeds];
  __shared__ uint32_t srev[kGWarps][kReadWords];  // the read's codes, first code in the high bits, 0 after its end
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int nseeds = gs.n;
  const int cap = go.warp_cap;
  int32_t* pos = sm + (size_t)w * gather_warp_words(cap);
  uint16_t* claims = reinterpret_cast<uint16_t*>(pos + ((cap + 31) & ~31));
  uint8_t* mark = reinterpret_cast<uint8_t*>(claims);  // item + 1 at the first position of an item, 0 elsewhere
  int2* item = reinterpret_cast<int2*>(claims + 2 * gather_half_words(cap));  // map offset - slot, read position | seed << 16
  uint16_t* undecided = reinterpret_cast<uint16_t*>(item);
  if (threadIdx.x == 0) s_nruns = 0;
  __syncthreads();
  if (threadIdx.x < nseeds) {
    s_first[threadIdx.x] = ix.first[threadIdx.x];
    s_map[threadIdx.x] = ix.map[threadIdx.x];
    sspan[threadIdx.x] = gs.s[threadIdx.x].span;
    if (gs.s[threadIdx.x].span <= 32) atomicMax(&s_nruns, make_runs(gs.s[threadIdx.x], runs[threadIdx.x]));
  }
  __syncthreads();
  const int nruns = s_nruns;
  int32_t* so = soff[w];
  uint32_t* rv = srev[w];
  unsigned long long lookups = 0, positions = 0;
  for (;;) {
  unsigned long long k0 = 0;
  if (lane == 0) k0 = atomicAdd(go.cursor, (unsigned long long)go.reads_per_steal);
  k0 = __shfl_sync(0xffffffffu, k0, 0);
  if ((int64_t)k0 >= rd.n) break;
  const int64_t kend = (int64_t)k0 + go.reads_per_steal < rd.n ? (int64_t)k0 + go.reads_per_steal : rd.n;
  for (int64_t kr = (int64_t)k0; kr < kend; ++kr) {
    const int64_t r = rd.order ? (int64_t)rd.order[kr] : kr;
    const int L = rd.lengths[r];
    const uint8_t* src = rd.codes + r * rd.cstride;
    {  // the read's packed codes into shared memory, and the item offsets of the seeds
      const int nb = (L + 3) >> 2, nw = (L + 15) >> 4;
      for (int k = lane; k < nw + 2; k += 32) {
        uint32_t x = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (4 * k + b < nb) x |= (uint32_t)src[4 * k + b] << (8 * b);
        const int left = L - 16 * k;  // codes of this word
        if (left < 16) x &= left > 0 ? (1u << (2 * left)) - 1u : 0u;
        rv[k] = reverse_codes(x);
      }
      const int np = lane < nseeds ? seed_npos(gs.s[lane], L) : 0;
      const int incl = warp_incl_scan(np);
      if (lane <= nseeds) so[lane] = incl - np;
      __syncwarp();
    }
    const int T = so[nseeds];
    int H = 0;
    int32_t vmin = kEmptySlot, v1 = kEmptySlot;  // v1: a read of at most 32 positions, one per lane
    // a read with more positions than the warp holds is only counted from there on and goes to
    // the block kernel with its count (its lookups and positions are counted there)
    for (int r0 = 0; r0 < T; r0 += 32 * kItems) {
      // every lane looks up its items (all key-table loads in flight together) ...
      int a[kItems], cnt[kItems], info[kItems];
#pragma unroll
      for (int m = 0; m < kItems; ++m) {
        const int it = r0 + m * 32 + lane;
        a[m] = 0; cnt[m] = 0; info[m] = 0;
        if (it < T) {
          int si = 0;
          while (it >= so[si + 1]) ++si;
          int rp = it - so[si];
          if (gs.s[si].n_positions) rp = gs.s[si].positions[rp];
          if (rp >= 0 && rp < L) {
            uint32_t key = 0;
            if (sspan[si] <= 32) {
              const uint32_t* q = rv + (rp >> 4);
              const int sh = 2 * (rp & 15);
              const uint64_t win = (uint64_t)__funnelshift_l(q[1], q[0], sh) << 32 | __funnelshift_l(q[2], q[1], sh);
#pragma unroll 4
              for (int c = 0; c < nruns; ++c) {
                const uint2 R = runs[si].r[c];
                key |= (uint32_t)(win >> R.x) & R.y;
              }
            } else {
              key = read_key(gs.s[si], src, L, rp);
            }
            a[m] = __ldg(s_first[si] + key);
            cnt[m] = __ldg(s_first[si] + key + 1) - a[m];
            info[m] = rp | si << 16;
          }
        }
      }
      // ... then one scan places all of them ...
      int tot = 0;
#pragma unroll
      for (int m = 0; m < kItems; ++m) tot += cnt[m];
      const int incl = warp_incl_scan(tot);
      const int n = __shfl_sync(0xffffffffu, incl, 31);  // positions of this round
      const int H0 = H;
      H += n;
      if (H > cap) continue;  // uniform over the warp: counting only
      if (n == 0) continue;
      for (int k = lane; 4 * k < n; k += 32) reinterpret_cast<uint32_t*>(mark)[k] = 0;
      __syncwarp();
      int dst = incl - tot;
#pragma unroll
      for (int m = 0; m < kItems; ++m) {
        if (cnt[m] > 0) {
          mark[dst] = (uint8_t)(lane * kItems + m + 1);
          item[lane * kItems + m] = make_int2(a[m] - dst, info[m]);
          dst += cnt[m];
        }
      }
      __syncwarp();
      // ... and the positions are spread over the lanes: position s belongs to the last item marked
      // at or before it
      int carry = 0;
      for (int s0 = 0; s0 < n; s0 += 32 * kChunks) {
        int32_t v[kChunks];
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          const int s = s0 + 32 * c + lane;
          v[c] = kEmptySlot;
          if (s0 + 32 * c < n) {  // uniform
            const int mk = s < n ? mark[s] : 0;
            const unsigned b = __ballot_sync(0xffffffffu, mk != 0) & (lt | (1u << lane));
            const int own = __shfl_sync(0xffffffffu, mk, b ? 31 - __clz(b) : lane);
            const int it = b ? own - 1 : carry;
            carry = __shfl_sync(0xffffffffu, it, 31);
            if (s < n) {
              const int2 e = item[it];
              v[c] = __ldg(s_map[e.y >> 16] + e.x + s) - (e.y & 0xffff);
            }
          }
        }
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          const int s = s0 + 32 * c + lane;
          vmin = min(vmin, v[c]);
          if (c == 0 && s0 == 0) v1 = v[0];
          if (s < n) pos[H0 + s] = v[c];
        }
      }
      __syncwarp();
    }
    if (H > cap) {
      if (lane == 0) {
        if (H <= kSmallGatherCap) {
          const int k = atomicAdd(go.big_count + 2, 1);
          go.small_list[k] = (int32_t)r;
          go.small_h[k] = H;
        } else {
          const int k = atomicAdd(go.big_count, 1);
          go.big_list[k] = (int32_t)r;
          go.big_h[k] = H;
        }
      }
      __syncwarp();
      continue;
    }
    positions += (unsigned long long)H;
    lookups += (unsigned long long)T;
    if (H == 0) continue;
    // the distinct diagonals to the flat list; the smallest is dropped when it is not above -I
    // (run.c:617, :648)
    vmin = __reduce_min_sync(0xffffffffu, vmin);
    const int32_t drop = vmin <= -I ? vmin : kEmptySlot;
    if (H <= 32) {
      if (T > 32 * kItems) v1 = lane < H ? pos[lane] : kEmptySlot;  // more than one round
      const unsigned peers = __match_any_sync(0xffffffffu, v1);
      const unsigned m = __ballot_sync(0xffffffffu, v1 != kEmptySlot && v1 != drop && (peers & lt) == 0);
      const int64_t base = reserve(go, __popc(m));
      if (base >= 0 && ((m >> lane) & 1u)) {
        const int64_t o = base + __popc(m & lt);
        go.fr[o] = (int32_t)r;
        go.fd[o] = v1;
      }
    } else {
      const int U = warp_distinct(pos, H, claims, cap, undecided) - (drop != kEmptySlot ? 1 : 0);
      int64_t o = reserve(go, U);
      if (o >= 0) {
        for (int k0 = 0; k0 < H; k0 += 32) {
          const int32_t v = k0 + lane < H ? pos[k0 + lane] : kEmptySlot;
          const bool keep = v != kEmptySlot && v != drop;
          const unsigned m = __ballot_sync(0xffffffffu, keep);
          if (keep) {
            go.fr[o + __popc(m & lt)] = (int32_t)r;
            go.fd[o + __popc(m & lt)] = v;
          }
          o += __popc(m);
        }
      }
    }
    __syncwarp();
  }
  }
  if (lane == 0) {  // both counts are the same in every lane of the warp
    atomicAdd(&go.counters[3], lookups);
    atomicAdd(&go.counters[4], positions);
  }
}

// One block per read of the list, for reads with more index positions than a warp holds: the
// positions go to a block-private slice of a global buffer (scratch: 2 * cap words per block,
// its working set small enough to stay in L2), then a bucket sort without comparisons across
// buckets: min / max, buckets of equal power-of-two width over [min, max] (about 8 values each,
// so that bucket order is value order), counted and scattered with shared atomics, then every
// thread insertion-sorts its buckets, dropping repeated values on the way.  The surviving
// diagonals are appended in order; the smallest is dropped when it is not above -I
// (run.c:617, :648).  Reads with more than `cap` positions are appended to (huge_list,
// huge_h) for a second launch with a larger cap.  The grid is persistent: blocks take the next
// read of the list from `cursor` (zeroed), list_count read on the device when given.
constexpr int kBT = 512;              // threads of a block-gather block
constexpr int kMaxBuckets = 4096;
constexpr int kSmallCap = kSmallGatherCap;  // a read with at most this many positions sorts in shared memory

// exclusive scan of a[0..n) in place (n <= kMaxBuckets, every thread of the block); the total
__device__ __forceinline__ int block_excl_scan(int32_t* a, int n, int* wtot) {
  constexpr int per = kMaxBuckets / kBT;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b0 = threadIdx.x * per;
  int loc = 0;
#pragma unroll
  for (int k = 0; k < per; ++k)
    if (b0 + k < n) loc += a[b0 + k];
  const int incl = warp_incl_scan(loc);
  if (lane == 31) wtot[w] = incl;
  __syncthreads();
  int before = 0, tot = 0;
  for (int q = 0; q < kBT / 32; ++q) {
    if (q < w) before += wtot[q];
    tot += wtot[q];
  }
  int run = before + incl - loc;
#pragma unroll
  for (int k = 0; k < per; ++k)
    if (b0 + k < n) {
      const int v = a[b0 + k];
      a[b0 + k] = run;
      run += v;
    }
  __syncthreads();
  return tot;
}

// SMEM: the slices in dynamic shared memory (every read of the list has at most kSmallCap
// positions).  Without it a launch keeps its shared memory small: the L1 cache shares that
// storage, and the global slices of reads with many positions live off it.
template <bool SMEM>
__global__ void __launch_bounds__(kBT) gather_block_kernel(ReadsDev rd, IndexView ix, int I, const int32_t* __restrict__ list,
                                                           const int32_t* __restrict__ list_h,
                                                           const int32_t* __restrict__ list_count, int64_t nlist,
                                                           GatherOut go, int32_t* __restrict__ scratch, int cap,
                                                           unsigned long long* cursor, int32_t* huge_list, int32_t* huge_h,
                                                           int32_t* huge_count, const __grid_constant__ SeedSet gs) {
  __shared__ int32_t cnt[kMaxBuckets];   // per bucket: count, start, then end
  __shared__ int32_t uoff[kMaxBuckets];  // per bucket: distinct values, then their offset
  __shared__ int wtot[kBT / 32];
  __shared__ int s_read, s_H;
  __shared__ int32_t s_min, s_max;
  __shared__ unsigned long long s_base;
  __shared__ __align__(16) uint8_t srd[kReadBytes];
  extern __shared__ int32_t dsm[];  // 2 * kSmallCap: the slices of a read with few positions
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int32_t* const Ag = scratch + (int64_t)blockIdx.x * 2 * cap;  // the block's slices in global memory
  int32_t* const Bg = Ag + cap;
  const int64_t n = list_count ? (int64_t)*list_count : nlist;
  unsigned long long lookups = 0, positions = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long k = atomicAdd(cursor, 1ull);
      s_read = (int64_t)k < n ? list[k] : -1;
      s_H = (int64_t)k < n ? list_h[k] : 0;
      s_min = 0x7fffffff;
      s_max = (int32_t)0x80000000;
    }
    __syncthreads();
    const int r = s_read;
    if (r < 0) break;
    const int L = rd.lengths[r];
    {
      const uint8_t* src = rd.codes + (int64_t)r * rd.cstride;
      const int nbytes = (L + 3) >> 2;
      for (int b = threadIdx.x; b < kReadBytes; b += kBT) srd[b] = b < nbytes ? src[b] : 0;
    }
    __syncthreads();
    // the read's position count came with it (the warp gather counted it), so a read above
    // `cap` loads none of its positions here
    int T = 0;
    for (int si = 0; si < gs.n; ++si) T += seed_npos(gs.s[si], L);
    const int H = s_H;
    if (H > cap) {
      if (threadIdx.x == 0) {
        const int k = atomicAdd(huge_count, 1);
        huge_list[k] = r;
        huge_h[k] = H;
      }
      __syncthreads();
      continue;
    }
    lookups += (unsigned long long)T;
    positions += (unsigned long long)H;
    if (H == 0) {
      __syncthreads();
      continue;
    }
    __syncthreads();  // every thread has read s_H
    if (threadIdx.x == 0) s_H = 0;
    __syncthreads();
    // the rest of the read, compiled twice: slices in shared memory (a read with few positions)
    // or in the block's global slices, each with plain shared or global memory operations
    auto per_read = [&](auto in_shared) {
      constexpr bool SMALL = decltype(in_shared)::value;
      int32_t* const A = SMALL ? dsm : Ag;
      int32_t* const B = SMALL ? dsm + kSmallCap : Bg;
      // gather: every (seed, read position) item's CSR range, placed by a block scan; the range
      // of the values is taken on the way
      int32_t vmin = 0x7fffffff, vmax = (int32_t)0x80000000;
      auto put = [&](int k, int32_t v) {
        vmin = min(vmin, v);
        vmax = max(vmax, v);
        A[k] = v;
      };
      for (int si = 0; si < gs.n; ++si) {
        const int np = seed_npos(gs.s[si], L);
        const int32_t* first = ix.first[si];
        const int32_t* mp = ix.map[si];
        for (int t0 = 0; t0 < np; t0 += kBT) {
          int a, c, rp;
          item_lookup(first, gs.s[si], t0 + threadIdx.x, srd, L, a, c, rp);
          const int incl = warp_incl_scan(c);
          if (lane == 31) wtot[w] = incl;
          __syncthreads();
          int before = 0, tot = 0;
          for (int q = 0; q < kBT / 32; ++q) {
            if (q < w) before += wtot[q];
            tot += wtot[q];
          }
          const int dst = s_H + before + incl - c;
          if (c <= 8) {
            for (int u = 0; u < c; ++u) put(dst + u, __ldg(mp + a + u) - rp);
          }
          unsigned bm = __ballot_sync(0xffffffffu, c > 8);  // long lists: the warp copies each
          while (bm) {
            const int j = __ffs(bm) - 1;
            bm &= bm - 1;
            const int aj = __shfl_sync(0xffffffffu, a, j), cj = __shfl_sync(0xffffffffu, c, j);
            const int dj = __shfl_sync(0xffffffffu, dst, j), rj = __shfl_sync(0xffffffffu, rp, j);
            for (int u = lane; u < cj; u += 32) put(dj + u, __ldg(mp + aj + u) - rj);
          }
          __syncthreads();
          if (threadIdx.x == 0) s_H += tot;
          __syncthreads();
        }
      }
      // range
      vmin = __reduce_min_sync(0xffffffffu, vmin);
      vmax = __reduce_max_sync(0xffffffffu, vmax);
      if (lane == 0) {
        atomicMin(&s_min, vmin);
        atomicMax(&s_max, vmax);
      }
      __syncthreads();
      vmin = s_min;
      const uint32_t range = (uint32_t)s_max - (uint32_t)vmin;
      int nb = 1;
      while (nb < kMaxBuckets && nb * 8 < H) nb <<= 1;
      int shift = 0;
      while ((range >> shift) >= (uint32_t)nb) ++shift;
      for (int b = threadIdx.x; b < nb; b += kBT) cnt[b] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < H; i += kBT) atomicAdd(&cnt[((uint32_t)A[i] - (uint32_t)vmin) >> shift], 1);
      __syncthreads();
      block_excl_scan(cnt, nb, wtot);
      for (int i = threadIdx.x; i < H; i += kBT) {
        const int32_t v = A[i];
        B[atomicAdd(&cnt[((uint32_t)v - (uint32_t)vmin) >> shift], 1)] = v;
      }
      __syncthreads();  // cnt[b] is now the end of bucket b
      for (int b = threadIdx.x; b < nb; b += kBT) {
        const int s0 = b ? cnt[b - 1] : 0, e = cnt[b];
        int u = 0;
        for (int x = s0; x < e; ++x) {  // insertion into the sorted distinct prefix B[s0, s0 + u)
          const int32_t t = B[x];
          int y = u - 1;
          while (y >= 0 && B[s0 + y] > t) --y;
          if (y >= 0 && B[s0 + y] == t) continue;
          for (int z = u - 1; z > y; --z) B[s0 + z + 1] = B[s0 + z];
          B[s0 + y + 1] = t;
          ++u;
        }
        uoff[b] = u;
      }
      __syncthreads();
      const int U = block_excl_scan(uoff, nb, wtot);
      for (int b = threadIdx.x; b < nb; b += kBT) {
        const int s0 = b ? cnt[b - 1] : 0, o = uoff[b];
        const int u = (b + 1 < nb ? uoff[b + 1] : U) - o;
        for (int k = 0; k < u; ++k) A[o + k] = B[s0 + k];
      }
      __syncthreads();
      const int drop = A[0] <= -I ? 1 : 0;  // the first diagonal must exceed -I (run.c:617, :648)
      const int Uo = U - drop;
      if (threadIdx.x == 0) s_base = Uo ? atomicAdd(&go.counters[7], (unsigned long long)Uo) : 0ull;
      __syncthreads();
      const unsigned long long base = s_base;
      if ((int64_t)(base + Uo) > go.cap) {
        if (threadIdx.x == 0) atomicExch(&go.counters[8], 1ull);
      } else {
        for (int k = threadIdx.x; k < Uo; k += kBT) {
          go.fr[base + k] = r;
          go.fd[base + k] = A[k + drop];
        }
      }
    };
    if constexpr (SMEM) per_read(std::true_type{});
    else per_read(std::false_type{});
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    atomicAdd(&go.counters[3], lookups);
    atomicAdd(&go.counters[4], positions);
  }
}

void launch_gather_fused(const ReadsDev& rd, const IndexView& ix, int I, const GatherOut& go, const SeedSet& seeds,
                         cudaStream_t st) {
  if (rd.n <= 0) return;
  set_smem_attribute_once(reinterpret_cast<const void*>(gather_fused_kernel), kGWarps * gather_warp_words(kMaxWarpCap) * 4);
  const size_t smem = (size_t)kGWarps * gather_warp_words(go.warp_cap) * sizeof(int32_t);
  const int64_t per_block = (int64_t)kGWarps * go.reads_per_steal;
  const int64_t blocks = std::min<int64_t>((rd.n + per_block - 1) / per_block,
                                          resident_grid(gather_fused_kernel, kGWarps * 32, smem));
  gather_fused_kernel<<<(unsigned)blocks, kGWarps * 32, smem, st>>>(rd, ix, I, go, seeds);
}

constexpr size_t kBlockGatherSmem = 2 * kSmallCap * sizeof(int32_t);

int64_t gather_block_grid(bool smem) {
  if (!smem) return resident_grid(gather_block_kernel<false>, kBT, 0);
  set_smem_attribute_once(reinterpret_cast<const void*>(gather_block_kernel<true>), (int)kBlockGatherSmem);
  return resident_grid(gather_block_kernel<true>, kBT, kBlockGatherSmem);
}

void launch_gather_block(const ReadsDev& rd, const IndexView& ix, int I, const int32_t* list, const int32_t* list_h,
                         int64_t nlist, const int32_t* nlist_dev, const GatherOut& go, int32_t* scratch, int cap,
                         int64_t grid, unsigned long long* cursor, int32_t* huge_list, int32_t* huge_h,
                         int32_t* huge_count, bool smem, const SeedSet& seeds, cudaStream_t st) {
  if (nlist <= 0 || grid <= 0) return;
  if (smem) {
    set_smem_attribute_once(reinterpret_cast<const void*>(gather_block_kernel<true>), (int)kBlockGatherSmem);
    gather_block_kernel<true><<<(unsigned)grid, kBT, kBlockGatherSmem, st>>>(
        rd, ix, I, list, list_h, nlist_dev, nlist, go, scratch, cap, cursor, huge_list, huge_h, huge_count, seeds);
  } else {
    gather_block_kernel<false><<<(unsigned)grid, kBT, 0, st>>>(rd, ix, I, list, list_h, nlist_dev, nlist, go, scratch,
                                                               cap, cursor, huge_list, huge_h, huge_count, seeds);
  }
}

}  // namespace sg
