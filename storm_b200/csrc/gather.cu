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
// block-per-read kernel (below), which appends ascending diagonals.
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

constexpr int kGWarps = 4;
// Reads per steal (GatherOut.reads_per_steal, 4 by default): the grid is the resident set, and
// every warp takes the next reads_per_steal reads (in the order of rd.order, or of the batch) from a work cursor until none is left, so
// reads with many index positions balance out, and warps append their candidates in close to
// read order: a batch whose reads are grouped by length gives a candidate list grouped by
// length, which the filter needs to keep one read length per SM.
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

void launch_gather_fused(const ReadsDev& rd, const IndexView& ix, int I, const GatherOut& go, const SeedSet& seeds,
                         cudaStream_t st) {
  if (rd.n <= 0) return;
  set_smem_attribute_once(reinterpret_cast<const void*>(gather_fused_kernel), kGWarps * gather_warp_words(kMaxWarpCap) * 4);
  const size_t smem = (size_t)kGWarps * gather_warp_words(go.warp_cap) * sizeof(int32_t);
  // a batch of few reads is spread over the SMs first: a block per read, and no more reads per steal
  // than leave every resident warp a turn (16 reads of 50 bp, one strand: 15 us, with 4 reads per steal 40)
  const int64_t resident = resident_grid(gather_fused_kernel, kGWarps * 32, smem);
  GatherOut g = go;
  g.reads_per_steal = (int)std::clamp<int64_t>(rd.n / (resident * kGWarps), 1, go.reads_per_steal);
  const int64_t blocks = std::min<int64_t>(rd.n, resident);
  gather_fused_kernel<<<(unsigned)blocks, kGWarps * 32, smem, st>>>(rd, ix, I, g, seeds);
}

// ------------------------------------------------------------------ reads with many positions

// One block per read of a list, for reads above the warp gather's bucket: a bucket sort without
// comparisons across buckets.  Buckets of equal power-of-two width (bucket order is value order), about
// 8 values each, counted and scattered with shared atomics; every thread then sorts its buckets,
// dropping repeated values, and the surviving diagonals are appended in order; the smallest is dropped
// when it is not above -I (run.c:617, :648).  The positions are read from the index once to be
// counted and once to be scattered straight into their buckets, so that one copy of them is held and
// not two.  The grid is persistent: blocks take the next read of the list from `cursor` (zeroed),
// list_count read on the device when given.
//   * kSmall, up to kSmallGatherCap positions: the diagonals in shared memory, buckets over their range,
//     several blocks per SM.
//   * kLarge, up to kSortGatherCap positions: buckets over the whole sequence, at most 2^16 codes wide, so
//     that 16 bits hold a diagonal's place in its bucket and 65,535 of them fit one SM's shared memory
//     (a 150-bp read meets 50,000 positions in a repeat-rich 100 Mbp genome under three w10 seeds).
//     Sequences too long for that (2^29 codes) go to (huge_list, huge_h), as do reads with more.
//   * kHuge, up to `cap` positions: as kSmall with the diagonals in a slice of global memory (scratch: cap
//     words per block) and more buckets; above cap to (huge_list, huge_h) for a launch with larger slices.
// What bounds it is the latency of shared memory in the buckets and of the index passes; with two
// global slices per block (L2-resident), insertion sorts in them and the position lists copied one by
// one, the same reads took 11.1 ms where this takes 4.3 ms (4,000 mixed reads, both strands).

constexpr int kReadBytes = STORMGPU_MAX_READ_LEN / 4 + 16;

// exclusive scan of a[0..n) in place, n <= NB, by every thread of the block; the total
template <int THREADS, int NB, class T>
__device__ __forceinline__ int sort_excl_scan(T* a, int n, int* wtot) {
  constexpr int per = NB / THREADS;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b0 = threadIdx.x * per;
  int loc = 0;
#pragma unroll
  for (int k = 0; k < per; ++k)
    if (b0 + k < n) loc += a[b0 + k];
  const int incl = warp_incl_scan(loc);
  if (lane == 31) wtot[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int t = lane < THREADS / 32 ? wtot[lane] : 0;
    const int i = warp_incl_scan(t);
    if (lane < THREADS / 32) wtot[lane] = i;
  }
  __syncthreads();
  int run = (w ? wtot[w - 1] : 0) + incl - loc;
  const int tot = wtot[THREADS / 32 - 1];
#pragma unroll
  for (int k = 0; k < per; ++k)
    if (b0 + k < n) {
      const int v = a[b0 + k];
      a[b0 + k] = (T)run;
      run += v;
    }
  __syncthreads();
  return tot;
}

// The items of a read, THREADS at a time, in shared memory, and body(place, diagonal) for every one of
// its positions, g lanes per item.
template <int THREADS>
struct SortItems {
  int32_t off[THREADS];      // map offset
  int32_t at[THREADS + 32];  // place of the first position; at[THREADS]: their number
  int32_t info[THREADS];     // read position | seed << 16
  int wtot[32];
};

template <int THREADS, class Body>
__device__ __forceinline__ void each_position(SortItems<THREADS>& it, const IndexView& ix, const SeedSet& gs,
                                              const uint8_t* srd, int L, int T, int H, Body body) {
  // lanes per item: about a third of an item's positions
  const int g = H >= 64 * T ? 32 : H >= 16 * T ? 8 : 4;
  const int sub = threadIdx.x & (g - 1), grp = threadIdx.x / g, ngrp = THREADS / g;
  int H0 = 0;
  for (int t0 = 0; t0 < T; t0 += THREADS) {
    int t = t0 + (int)threadIdx.x, si = 0;
    int a = 0, c = 0, rp = 0;
    if (t < T) {
      for (; si < gs.n - 1; ++si) {
        const int np = seed_npos(gs.s[si], L);
        if (t < np) break;
        t -= np;
      }
      item_lookup(ix.first[si], gs.s[si], t, srd, L, a, c, rp);
    }
    it.off[threadIdx.x] = a;
    it.info[threadIdx.x] = c > 0 ? rp | si << 16 : 0;
    it.at[threadIdx.x] = c;
    __syncthreads();
    const int tot = sort_excl_scan<THREADS, THREADS>(it.at, THREADS, it.wtot);
    if (threadIdx.x == 0) it.at[THREADS] = tot;
    __syncthreads();
    const int ni = min(THREADS, T - t0);
    for (int q = grp; q < ni; q += ngrp) {
      const int o = it.at[q], cq = it.at[q + 1] - o;
      const int e = it.info[q], rq = e & 0xffff;
      const int32_t* mp = ix.map[e >> 16] + it.off[q];
      for (int u = sub; u < cq; u += 4 * g) {
        int32_t v[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) v[x] = u + x * g < cq ? __ldg(mp + u + x * g) : 0;
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (u + x * g < cq) body(H0 + o + u + x * g, v[x] - rq);
      }
    }
    H0 += tot;
    __syncthreads();
  }
}

// Batcher's odd-even merge sort of N registers, every index a constant.
template <int N>
__device__ __forceinline__ void sort_network(int32_t (&v)[N]) {
#pragma unroll
  for (int p = 1; p < N; p <<= 1)
#pragma unroll
    for (int k = p; k >= 1; k >>= 1)
#pragma unroll
      for (int j = k % p; j + k < N; j += 2 * k)
#pragma unroll
        for (int i = 0; i < k; ++i)
          if (i + j + k < N && (i + j) / (2 * p) == (i + j + k) / (2 * p)) {
            const int32_t x = v[i + j], y = v[i + j + k];
            v[i + j] = min(x, y);
            v[i + j + k] = max(x, y);
          }
}

// Sorts and de-duplicates the N - or less - values B[s0, s0 + n) in registers; the number of distinct
// ones.
template <int N, class V>
__device__ __forceinline__ int sort_bucket_regs(V* B, int s0, int n) {
  int32_t v[N];
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = k < n ? (int32_t)B[s0 + k] : kEmptySlot;
  sort_network<N>(v);
  int u = 0;
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (v[k] != kEmptySlot && (k == 0 || v[k] != v[k > 0 ? k - 1 : 0])) B[s0 + u++] = (V)v[k];
  return u;
}

// Sorts and de-duplicates B[s0, e) (one thread); the number of distinct values.  Up to 16 values go
// through a sorting network, the same instructions in every lane (insertion, whose steps differ from
// lane to lane, ran 13 of 32 lanes: 576 against 441 us for 1,000 mixed reads, one strand).
template <class V>
__device__ __forceinline__ int sort_bucket(V* B, int s0, int e) {
  const int n = e - s0;
  if (n <= 1) return n;
  if (n <= 8) return sort_bucket_regs<8>(B, s0, n);
  if (n <= 16) return sort_bucket_regs<16>(B, s0, n);
  int u = 0;
  for (int x = s0; x < e; ++x) {  // insertion into the sorted distinct prefix B[s0, s0 + u)
    const V t = B[x];
    int y = u - 1;
    while (y >= 0 && B[s0 + y] > t) --y;
    if (y >= 0 && B[s0 + y] == t) continue;
    for (int z = u - 1; z > y; --z) B[s0 + z + 1] = B[s0 + z];
    B[s0 + y + 1] = t;
    ++u;
  }
  return u;
}

enum SortKind { kSmall, kLarge, kHuge };

template <SortKind KIND>
struct SortConfig {
  static constexpr int CAP = KIND == kSmall ? kSmallGatherCap : KIND == kLarge ? kSortGatherCap : 0;  // in shared memory
  static constexpr int THREADS = KIND == kSmall ? 256 : 1024;
  static constexpr int NB = KIND == kSmall ? 1024 : KIND == kLarge ? 8192 : 16384;
  using V = typename std::conditional<KIND == kLarge, uint16_t, int32_t>::type;  // a diagonal, or its place in its bucket
  using U = typename std::conditional<KIND == kHuge, int32_t, uint16_t>::type;   // an offset in the read's list
  struct Smem {
    int32_t cnt[NB];  // per bucket: count, start, then end
    SortItems<THREADS> items;
    U uoff[NB];  // per bucket: distinct values, then their offset
    V B[CAP > 0 ? CAP : 1];
  };
};
static_assert(kSortGatherCap < 65536 && sizeof(SortConfig<kLarge>::Smem) <= 226 * 1024 &&
                  sizeof(SortConfig<kHuge>::Smem) <= 226 * 1024,
              "16-bit offsets, shared memory of an SM");

template <SortKind KIND>
__global__ void __launch_bounds__(SortConfig<KIND>::THREADS) gather_sort_kernel(
    ReadsDev rd, IndexView ix, int I, int64_t n_codes, const int32_t* __restrict__ list, const int32_t* __restrict__ list_h,
    const int32_t* __restrict__ list_count, int64_t nlist, GatherOut go, int32_t* __restrict__ scratch, int cap,
    unsigned long long* cursor, int32_t* huge_list, int32_t* huge_h, int32_t* huge_count,
    const __grid_constant__ SeedSet gs) {
  using Cf = SortConfig<KIND>;
  using V = typename Cf::V;
  constexpr int THREADS = Cf::THREADS, NB = Cf::NB;
  extern __shared__ __align__(16) uint8_t dsm[];
  typename Cf::Smem& S = *reinterpret_cast<typename Cf::Smem*>(dsm);
  V* const B = KIND == kHuge ? reinterpret_cast<V*>(scratch + (int64_t)blockIdx.x * cap) : S.B;
  __shared__ int s_read, s_H, s_drop;
  __shared__ int32_t s_min, s_max;
  __shared__ unsigned long long s_base;
  __shared__ __align__(16) uint8_t srd[kReadBytes];
  const int64_t n = list_count ? (int64_t)*list_count : nlist;
  // the large form's buckets: diagonals from -kMaxReadLen to n_codes
  int shift_all = 0;
  while (((n_codes + STORMGPU_MAX_READ_LEN) >> shift_all) >= NB) ++shift_all;
  unsigned long long lookups = 0, positions = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long k = atomicAdd(cursor, 1ull);
      s_read = (int64_t)k < n ? list[k] : -1;
      s_H = (int64_t)k < n ? list_h[k] : 0;
      s_min = 0x7fffffff;
      s_max = (int32_t)0x80000000;
      s_drop = 0;
    }
    __syncthreads();
    const int r = s_read, H = s_H;
    if (r < 0) break;
    if (H > (KIND == kHuge ? cap : Cf::CAP) || (KIND == kLarge && shift_all > 16)) {
      if (threadIdx.x == 0) {
        const int k = atomicAdd(huge_count, 1);
        huge_list[k] = r;
        huge_h[k] = H;
      }
      __syncthreads();
      continue;
    }
    const int L = rd.lengths[r];
    {
      const uint8_t* src = rd.codes + (int64_t)r * rd.cstride;
      const int nbytes = (L + 3) >> 2;
      for (int b = threadIdx.x; b < kReadBytes; b += THREADS) srd[b] = b < nbytes ? src[b] : 0;
    }
    int T = 0;
    for (int si = 0; si < gs.n; ++si) T += seed_npos(gs.s[si], L);
    lookups += (unsigned long long)T;
    positions += (unsigned long long)H;
    int nb = NB, shift = shift_all;
    int32_t vmin = -STORMGPU_MAX_READ_LEN;
    if constexpr (KIND != kLarge) {
      nb = 1;
      while (nb < NB && nb * 8 < H) nb <<= 1;
    }
    for (int b = threadIdx.x; b < nb; b += THREADS) S.cnt[b] = 0;
    __syncthreads();
    if constexpr (KIND != kLarge) {
      vmin = 0x7fffffff;
      int32_t vmax = (int32_t)0x80000000;
      each_position<THREADS>(S.items, ix, gs, srd, L, T, H, [&](int k, int32_t v) {
        vmin = min(vmin, v);
        vmax = max(vmax, v);
        B[k] = v;
      });
      vmin = __reduce_min_sync(0xffffffffu, vmin);
      vmax = __reduce_max_sync(0xffffffffu, vmax);
      if ((threadIdx.x & 31) == 0) {
        atomicMin(&s_min, vmin);
        atomicMax(&s_max, vmax);
      }
      __syncthreads();
      vmin = s_min;
      const uint32_t range = (uint32_t)s_max - (uint32_t)vmin;
      shift = 0;
      while ((range >> shift) >= (uint32_t)nb) ++shift;
      for (int i = threadIdx.x; i < H; i += THREADS) atomicAdd(&S.cnt[((uint32_t)B[i] - (uint32_t)vmin) >> shift], 1);
    } else {
      each_position<THREADS>(S.items, ix, gs, srd, L, T, H,
                             [&](int, int32_t v) { atomicAdd(&S.cnt[((uint32_t)v - (uint32_t)vmin) >> shift], 1); });
    }
    __syncthreads();
    sort_excl_scan<THREADS, NB>(S.cnt, nb, S.items.wtot);
    each_position<THREADS>(S.items, ix, gs, srd, L, T, H, [&](int, int32_t v) {
      const uint32_t x = (uint32_t)v - (uint32_t)vmin;
      B[atomicAdd(&S.cnt[x >> shift], 1)] = KIND != kLarge ? (V)v : (V)(x & ((1u << shift) - 1u));
    });
    // cnt[b] is now the end of bucket b
    for (int b = threadIdx.x; b < nb; b += THREADS)
      S.uoff[b] = (typename Cf::U)sort_bucket(B, b ? S.cnt[b - 1] : 0, S.cnt[b]);
    __syncthreads();
    const int U = sort_excl_scan<THREADS, NB>(S.uoff, nb, S.items.wtot);
    // bucket b: its first slot, the offset of its distinct values and their number; the diagonals
    auto bucket = [&](int b, int& s0, int& o, int& u) {
      s0 = b ? S.cnt[b - 1] : 0;
      o = S.uoff[b];
      u = (b + 1 < nb ? (int)S.uoff[b + 1] : U) - o;
    };
    auto value = [&](int b, int at) -> int32_t {
      return KIND != kLarge ? (int32_t)B[at] : (int32_t)((uint32_t)vmin + ((uint32_t)b << shift) + (uint32_t)B[at]);
    };
    for (int b = threadIdx.x; b < nb; b += THREADS) {  // the first diagonal must exceed -I (run.c:617, :648)
      int s0, o, u;
      bucket(b, s0, o, u);
      if (o == 0 && u > 0 && value(b, s0) <= -I) s_drop = 1;
    }
    __syncthreads();
    const int drop = s_drop, Uo = U - drop;
    if (threadIdx.x == 0) s_base = Uo > 0 ? atomicAdd(&go.counters[7], (unsigned long long)Uo) : 0ull;
    __syncthreads();
    const unsigned long long base = s_base;
    if ((int64_t)(base + Uo) > go.cap) {
      if (threadIdx.x == 0) atomicExch(&go.counters[8], 1ull);
    } else {
      for (int k = threadIdx.x; k < Uo; k += THREADS) go.fr[base + k] = r;
      for (int b = threadIdx.x; b < nb; b += THREADS) {
        int s0, o, u;
        bucket(b, s0, o, u);
        for (int k = 0; k < u; ++k)
          if (o + k >= drop) go.fd[base + o + k - drop] = value(b, s0 + k);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    atomicAdd(&go.counters[3], lookups);
    atomicAdd(&go.counters[4], positions);
  }
}

int64_t gather_huge_grid() {
  set_smem_attribute_once(reinterpret_cast<const void*>(gather_sort_kernel<kHuge>), (int)sizeof(SortConfig<kHuge>::Smem));
  return resident_grid(gather_sort_kernel<kHuge>, SortConfig<kHuge>::THREADS, sizeof(SortConfig<kHuge>::Smem));
}

template <SortKind KIND>
static void launch_sort(const ReadsDev& rd, const IndexView& ix, int I, int64_t n_codes, const GatherList& l,
                        const GatherOut& go, int32_t* scratch, int cap, int64_t max_grid, const SeedSet& seeds,
                        cudaStream_t st) {
  if (l.n <= 0 || max_grid <= 0) return;
  constexpr size_t smem = sizeof(typename SortConfig<KIND>::Smem);
  constexpr int threads = SortConfig<KIND>::THREADS;
  set_smem_attribute_once(reinterpret_cast<const void*>(gather_sort_kernel<KIND>), (int)smem);
  const int64_t grid = std::min({l.n, max_grid, resident_grid(gather_sort_kernel<KIND>, threads, smem)});
  gather_sort_kernel<KIND><<<(unsigned)grid, threads, smem, st>>>(rd, ix, I, n_codes, l.read, l.h, l.n_dev, l.n, go,
                                                                  scratch, cap, l.cursor, l.above, l.above_h,
                                                                  l.above_count, seeds);
}

void launch_gather_sort(const ReadsDev& rd, const IndexView& ix, int I, int64_t n_codes, const GatherList& l, bool small,
                        const GatherOut& go, const SeedSet& seeds, cudaStream_t st) {
  if (small) launch_sort<kSmall>(rd, ix, I, n_codes, l, go, nullptr, 0, INT64_MAX, seeds, st);
  else launch_sort<kLarge>(rd, ix, I, n_codes, l, go, nullptr, 0, INT64_MAX, seeds, st);
}

void launch_gather_huge(const ReadsDev& rd, const IndexView& ix, int I, int64_t n_codes, const GatherList& l,
                        int32_t* scratch, int cap, int64_t grid, const GatherOut& go, const SeedSet& seeds,
                        cudaStream_t st) {
  launch_sort<kHuge>(rd, ix, I, n_codes, l, go, scratch, cap, grid, seeds, st);
}

}  // namespace sg
