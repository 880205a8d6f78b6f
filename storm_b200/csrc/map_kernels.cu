// map_kernels.cu -- the kernels of one mapping pass (one reference sequence x one strand).
//
//  (hit gather: gather.cu; banded filter: sw_filter.cu; score bound: score_bound.cu)
//  align                                            banded DP + traceback (alignment.c:488-734): a thread per
//                                                   candidate in align_core.cuh, a warp here
//  replay                                           per-read top-4 update (run.c:664-691,
//                                                   hit_map.c:50-144)
#include "map_kernels.cuh"
#include "align_core.cuh"

namespace sg {

// ------------------------------------------------------------------------------ reads

__global__ void reverse_reads_kernel(ReadsDev in, const uint8_t* __restrict__ first_levels, int colour,
                                     uint8_t* __restrict__ rcodes, uint8_t* __restrict__ rlevels) {
  int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= in.n) return;
  const int L = in.lengths[r];
  const uint8_t* c = in.codes + r * in.cstride;
  uint8_t* rc = rcodes + r * in.cstride;
  for (int64_t b = 0; b < in.cstride; ++b) rc[b] = 0;
  // read__reverse (reads_data.c:9-35): nucleotide = reverse complement, colour = reverse
  for (int i = 0; i < L; ++i) {
    int v = code_at(c, i);
    if (!colour) v = 3 - v;
    int o = L - 1 - i;
    rc[o >> 2] |= (uint8_t)(v << ((o & 3) << 1));
  }
  if (in.levels) {
    const uint8_t* q = in.levels + r * in.lstride;
    uint8_t* rq = rlevels + r * in.lstride;
    for (int64_t b = 0; b < in.lstride; ++b) rq[b] = 0;
    if (!colour) {
      for (int i = 0; i < L; ++i) rq[i >> 2] |= (uint8_t)(code_at(q, L - 1 - i) << ((i & 3) << 1));
    } else {
      // quality__reverse_compressed, colour (read_quality.c:238-241)
      int fl = first_levels ? first_levels[r] : 3;
      rq[(L - 1) >> 2] |= (uint8_t)((fl & 3) << (((L - 1) & 3) << 1));
      for (int i = 0; i < L - 1; ++i) rq[i >> 2] |= (uint8_t)(code_at(q, L - 2 - i) << ((i & 3) << 1));
    }
  }
}

void launch_reverse_reads(const ReadsDev& in, const uint8_t* first_levels, int colour,
                          uint8_t* rcodes, uint8_t* rlevels, cudaStream_t st) {
  if (in.n <= 0) return;
  reverse_reads_kernel<<<(unsigned)((in.n + 127) / 128), 128, 0, st>>>(in, first_levels, colour, rcodes, rlevels);
}

__global__ void init_results_kernel(int64_t n, stormgpu_hit* __restrict__ hits, uint8_t* __restrict__ mapped) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * 4) return;
  stormgpu_hit h;
  h.score = kMinScore;
  h.ref_id = h.ref_start = h.ref_end = -1;
  h.read_start = h.read_end = -1;
  h.sense = 0;
  h.tb_len = 0;
  hits[t] = h;
  if ((t & 3) == 0) mapped[t >> 2] = 0;
}

void launch_init_results(int64_t n, stormgpu_hit* hits, uint8_t* mapped, uint8_t* tb, int64_t tbs,
                         cudaStream_t st) {
  if (n <= 0) return;
  init_results_kernel<<<(unsigned)((n * 4 + 255) / 256), 256, 0, st>>>(n, hits, mapped);
  cudaMemsetAsync(tb, 0, (size_t)(n * 4 * tbs), st);  // the 4n traceback rows are contiguous
}

// ------------------------------------------------------------------------------ align

// The packed nucleotide form has every band width up to 41 as a constant (the general form in local
// memory ran -i 5 at 50 GCUPS, a twentieth of the packed form's rate); the others the widths listed with them.
static const void* align_kernel_of(const ScoreParams& sp) {
  const int bw = 2 * sp.I + 1;
  const void* k = sp.packed == 2 ? align_unit_kernel(bw) : sp.packed ? align_packed_kernel(bw) : nullptr;
  return k ? k : align_general_kernel(bw, sp.colour);
}

int64_t align_workers(int64_t nslots, const ScoreParams& sp) {
  const int64_t g = resident_grid_of(align_kernel_of(sp), 128, 0) * 128;
  return std::min<int64_t>(g, (nslots + 127) / 128 * 128);
}

// ------------------------------------------------------------------------------ align, few slots

// The alignment of align_one by a warp per slot, for calls with so few slots that a thread each leaves
// the GPU idle while every thread walks its rows cell by cell: lane c holds cell c of the band and
// is at row i at time 2i + c, when the cell to its left (lane c - 1, same row) and the one above
// (lane c + 1, the row before) are one time step old.  The row maximum travels along with the row.
// Directions stay in shared memory (a byte per cell: direction, bit 2 the SNP adjustment), where lane
// 0 walks them back.  Every lane runs the same instructions in every step (those whose turn it is not
// discard the result).  2L + 2I + 1 steps of about 60 instructions, against L (2I + 1) cells of 25 to 40:
// 800 windows of 101 codes take 85 us at -i 15 where a thread each takes 127, 95 us in colours at -i 7
// against 290 (the whole call).  The chain of a step (shuffle, sums, state, next row's codes) is what
// bounds it: 31 % of the issue slots are taken with 5 warps an SM.
template <bool COLOUR>
__global__ void __launch_bounds__(32) align_wave_kernel(ReadsDev rd, ScoreParams sp, const uint8_t* __restrict__ genome,
                                                        const uint8_t* __restrict__ mask, int64_t slot0, int64_t nslots,
                                                        PassBuffers pb, int maxL) {
  extern __shared__ __align__(16) uint8_t wsm[];
  __shared__ uint8_t ctab[COLOUR ? kColourTable : 1];
  const int lane = threadIdx.x;
  const int64_t n = pb.npass_dev ? *pb.npass_dev : nslots;
  if (n > wave_slots(sp) || (int64_t)blockIdx.x >= n) return;
  const int I = sp.I, BW = 2 * I + 1;
  constexpr bool colour = COLOUR;
  int2* const pair_s = reinterpret_cast<int2*>(wsm);       // per read position: match and mismatch score
  uint8_t* const dir = wsm + sizeof(int2) * maxL;          // 32 per row
  uint8_t* const rc_s = dir + 32 * maxL;                   // per read position: code | level << 2
  uint8_t* const gc_s = rc_s + maxL;                       // per window position: code | masked << 2
  if (colour) {
    for (int k = lane; k < kColourTable; k += 32) ctab[k] = colour_step(k);
    __syncwarp();
  }
  const int mbest = sp.pair[0][3];
  unsigned long long rows = 0;
  for (int64_t s = blockIdx.x; s < n; s += gridDim.x) {
    const int64_t slot = slot0 + s;
    const int r = pb.p_read[slot];
    const int L = rd.lengths[r];
    const int64_t win = max(pb.p_diag[slot] - I, -sp.Is);  // run.c:667
    const uint8_t* rdc = rd.codes + (int64_t)r * rd.cstride;
    const uint8_t* rdq = rd.levels ? rd.levels + (int64_t)r * rd.lstride : nullptr;
    __syncwarp();
    for (int i = lane; i < L; i += 32) {
      const int q = rdq ? code_at(rdq, i) : 3;
      rc_s[i] = (uint8_t)(code_at(rdc, i) | q << 2);
      pair_s[i] = make_int2(sp.pair[0][q], sp.pair[1][q]);
    }
    for (int i = lane; i < L + 2 * I; i += 32)
      gc_s[i] = (uint8_t)(code_at(genome, win + i) | (code_at(mask, win + i) ? 4 : 0));
    __syncwarp();
    // row 0
    int sc = kMinScore, st = st_make(3, 0, 0, 0, 0);
    if (lane < BW) {
      const int x = rc_s[0], rc = x & 3, q = x >> 2, g = gc_s[lane], f = g & 3;
      int chk = 0;
      if (!(g & 4)) {
        chk = colour ? (rc ^ f) : 0;
        sc = sp.pair[colour ? (chk ? 1 : 0) : (rc != f)][q];
      }
      st = st_make(3, 0, chk, chk, (colour && chk) ? q : 0);
      dir[lane] = 3;
    }
    long long bound = 0x7fffffffLL;
    int best_possible = (colour ? (L - 2) : L) * mbest;
    int mol = kMinScore;  // of the row this lane was last at, its cells up to this lane's
    const int last_t = 2 * (L - 1) + BW - 1;
    const int border = st_make(3, I, 0, 0, 0);
    const bool first = lane == 0, last = lane == BW - 1, inband = lane < BW;
    int i = 1;  // the row this lane is at next, at time 2i + lane; its read and window codes
    int x = rc_s[min(1, L - 1)], g = gc_s[min(1 + lane, L + 2 * I - 1)];
    int2 pr = pair_s[min(1, L - 1)];
    for (int t = 2; t <= last_t; ++t) {
      int lsc = __shfl_up_sync(0xffffffffu, sc, 1), lst = __shfl_up_sync(0xffffffffu, st, 1);
      int tsc = __shfl_down_sync(0xffffffffu, sc, 1), tst = __shfl_down_sync(0xffffffffu, st, 1);
      int lmol = __shfl_up_sync(0xffffffffu, mol, 1);
      if (first) { lsc = kMinScore; lst = border; lmol = kMinScore; }
      if (last) { tsc = kMinScore; tst = border; }
      const bool now = inband && t == 2 * i + lane && i < L;
      const int rc = x & 3, q = x >> 2, f = g & 3;
      const bool masked = (g & 4) != 0;
      const int chk0 = colour && !masked ? rc ^ f : 0;
      const int s0 = masked ? kMinScore : rc != f ? pr.y : pr.x;
      int ms = s0, step = 0;
      if (colour) {
        step = ctab[(st >> 9) | (chk0 << 7) | (q << 9)];
        ms = (step & 0x80) && !masked && s0 < 0 ? -2 * s0 : s0;
      }
      const int cs = sc + ms;
      const int ts = tsc + (st_from(tst) == 2 ? sp.gap_ext : sp.gap_open);
      const int ls = lsc + (st_from(lst) == 1 ? sp.gap_ext : sp.gap_open);
      const bool top = st_ind(tst) < I && ts > cs;
      const int m1 = top ? ts : cs;
      const bool left = st_ind(lst) < I && ls > m1;
      const int score = left ? ls : m1;
      const int gst = left ? lst : tst;
      int gap = (left ? 1 : 2) | ((st_ind(gst) + 1) << 2);
      int cor = 3 | (st & 0x1FC);
      if (colour) {
        const bool fresh = st_fr(gst) > 1;
        const int ac = fresh ? st_ac(st) : chk0, fr = fresh ? st_fr(gst) - 1 : chk0 ? q : 0;
        gap |= ((st_chk(gst) ^ (left ? f : rc)) << 9) | (ac << 11) | (fr << 13);
        cor |= (step & 0x7F) << 9;
      }
      const bool corner = !top && !left;
      const int nst = corner ? cor : gap;
      if (now) {
        st = nst;
        sc = score;
        dir[32 * i + lane] = (uint8_t)((nst & 3) | (colour && corner && ms > 0 ? 4 : 0));
        mol = max(lmol, score);
        if (last) {  // the row is complete
          bound = min(bound, (long long)mol + best_possible);
          best_possible -= mbest;
        }
        ++i;
        const int in = min(i, L - 1);
        x = rc_s[in];
        pr = pair_s[in];
        g = gc_s[in + lane];
      }
    }
    __syncwarp();
    // the first of the largest cells of the last row
    const int top = __reduce_max_sync(0xffffffffu, lane < BW ? sc : kMinScore);
    const unsigned at = __ballot_sync(0xffffffffu, lane < BW && sc == top);
    const int bi = top > kMinScore ? L - 1 : -1, bc = top > kMinScore ? __ffs(at) - 1 : 0;
    const int32_t bnd = (int32_t)__shfl_sync(0xffffffffu, (int)bound, BW - 1);
    if (lane == 0) {
      const int bj = bi < 0 ? -1 : L - 1 + bc;
      int i0 = bi, j0 = bj, tl = 0;
      if (bi >= 0 && bnd >= sp.min_score && top > sp.min_score) {
        uint8_t* tb = pb.a_tb + slot * pb.tbs;
        uint8_t cur = 0;
        int c = bc, colr = 0;
        i = bi;
        while (i >= 0 && c >= 0 && c < BW) {
          const int d = dir[32 * i + c], from = d & 3, rc = rc_s[i] & 3, f = gc_s[i + c] & 3;
          i0 = i;
          j0 = i + c;
          int op;
          if (from == 2) op = 0xC | rc;
          else if (from == 1) op = 0x1;
          else if (rc == f) op = 0x3;
          else if (!colour || !(colr || ((d & 4) && i != 0 && i + c != 0))) op = 0x4 | rc;
          else { op = 0x8 | rc; colr ^= rc ^ f; }
          if (tl & 1) { cur |= (uint8_t)op; tb[tl >> 1] = cur; }
          else { cur = (uint8_t)(op << 4); tb[tl >> 1] = cur; }
          tl++;
          if (from == 2) { i--; c++; }
          else if (from == 1) { c--; }
          else { i--; }
        }
      }
      pb.a_score[slot] = top;
      pb.a_bound[slot] = bnd;
      pb.a_tblen[slot] = tl;
      pb.a_pos[slot * 4 + 0] = (int16_t)bi;
      pb.a_pos[slot * 4 + 1] = (int16_t)bj;
      pb.a_pos[slot * 4 + 2] = (int16_t)i0;
      pb.a_pos[slot * 4 + 3] = (int16_t)j0;
    }
    rows += (unsigned long long)L;
  }
  if (pb.cells && lane == 0 && rows) atomicAdd(pb.cells, rows * (unsigned long long)BW);
}

void launch_align_wave(const ReadsDev& r, const ScoreParams& sp, const uint8_t* genome, const uint8_t* mask,
                       int64_t slot0, int64_t nslots, PassBuffers& pb, int maxL, cudaStream_t st) {
  if (nslots <= 0) return;
  const size_t smem = (size_t)maxL * (33 + sizeof(int2)) + maxL + 2 * sp.I + 32;
  const int most = STORMGPU_MAX_READ_LEN * (34 + (int)sizeof(int2)) + 64;
  // passes enqueued ahead launch it for a whole list capacity
  const unsigned grid = (unsigned)std::min<int64_t>(nslots, wave_slots(sp));
  if (!grid) return;
  if (sp.colour) {
    set_smem_attribute_once(reinterpret_cast<const void*>(align_wave_kernel<true>), most);
    align_wave_kernel<true><<<grid, 32, smem, st>>>(r, sp, genome, mask, slot0, nslots, pb, maxL);
  } else {
    set_smem_attribute_once(reinterpret_cast<const void*>(align_wave_kernel<false>), most);
    align_wave_kernel<false><<<grid, 32, smem, st>>>(r, sp, genome, mask, slot0, nslots, pb, maxL);
  }
}

void launch_align(const ReadsDev& r, const ScoreParams& sp, const uint8_t* genome,
                  const uint8_t* mask, int64_t slot0, int64_t nslots, PassBuffers& pb,
                  cudaStream_t st) {
  if (nslots <= 0) return;
  const void* k = align_kernel_of(sp);
  // one slot per thread: few slots as warps on as many SMs as there are
  const int threads = !pb.cursor && nslots <= 148 * 64 ? 32 : 128;
  const unsigned blocks = (unsigned)(pb.cursor ? align_workers(nslots, sp) / 128 : (nslots + threads - 1) / threads);
  void* args[] = {(void*)&r, (void*)&sp, (void*)&genome, (void*)&mask, (void*)&slot0, (void*)&nslots, (void*)&pb};
  cudaLaunchKernel(k, dim3(blocks), dim3(threads), args, 0, st);  // errors surface at the caller's next check
}

// ------------------------------------------------------------------------------ replay

__device__ __forceinline__ int tbget(const uint8_t* t, int i) { return (t[i >> 1] >> ((i & 1) ? 0 : 4)) & 0xF; }

// process_read's acceptance (run.c:664-691) in the reference's order, with the
// threshold starting at -t for every (sequence, strand, read): aborted iff the bound is
// below the running threshold; accepted iff not aborted and score > threshold; then
// hit_map__update (hit_map.c:50-144) and threshold = max(threshold, 4th score).
//
// One warp per read: the lanes test 32 candidates at once against the threshold (few of a read's
// hundreds exceed it), lane 0 runs the update for those that do, on the read's four hits in shared
// memory, and the threshold it leaves is tested again.  Tracebacks are written once, at the end, from
// where each surviving hit came from.
//
// The warps go over a list of reads, those with candidates left (pb.active): slot_lists_kernel fills
// the first one, each round's replay the next, so that a round in which few reads have work costs a
// launch and no more.
//
// With rounds (pb.round_slots) the kernel replays the ranks its read's last selection covered and
// then selects the next ones: the ranks from there on whose score bound exceeds the threshold (all,
// without bounds), up to `take` of them (0: none left to select), appended to the next round's list;
// ranks passed over are marked as below every threshold.  Each round quadruples or so the ranks a
// read has behind it, and of those after them only about 4 per (ranks seen) can still enter the
// four hits, so nearly every later candidate is dropped by its bound alone.
constexpr int kReplayWarps = 4;

// hit_map__update for one accepted candidate on h[4] (src: where each hit's traceback is, -1 - row
// for a row already in place, else the slot).
__device__ __forceinline__ void hit_update(stormgpu_hit* h, int64_t* src, const PassBuffers& pb, const ScoreParams& sp,
                                           int64_t slot, int score, int ref_id, int sense) {
  const int win = max(pb.p_diag[slot] - sp.I, -sp.Is);
  const int bi = pb.a_pos[slot * 4 + 0], bj = pb.a_pos[slot * 4 + 1];
  const int i0 = pb.a_pos[slot * 4 + 2], j0 = pb.a_pos[slot * 4 + 3];
  int q;
  for (q = 0; q < 4 && h[q].ref_id != -1; ++q) {
    if (h[q].ref_id == ref_id && ((h[q].ref_start == win + j0 && h[q].read_start == i0) ||
                                  (h[q].ref_end == win + bj && h[q].read_end == bi))) {
      if (score > h[q].score) break;
      return;  // the same place with a score at least as high
    }
  }
  if (q == 4) q--;
  int i = q;
  while (i >= 0 && score > h[i].score) i--;
  if (i == 3) return;
  for (int j = q; j > i + 1; --j) {
    h[j] = h[j - 1];
    src[j] = src[j - 1];
  }
  stormgpu_hit nh;
  nh.score = score;
  nh.ref_id = ref_id;
  nh.ref_start = win + j0;
  nh.ref_end = win + bj;
  nh.read_start = (int16_t)i0;
  nh.read_end = (int16_t)bi;
  nh.sense = sense;
  nh.tb_len = pb.a_tblen[slot];
  h[i + 1] = nh;
  src[i + 1] = slot;
}

__device__ __forceinline__ void replay_read(int64_t r, const ScoreParams& sp, int ref_id, int sense, const PassBuffers& pb,
                                            int take, stormgpu_hit* __restrict__ hits, uint8_t* __restrict__ tbo,
                                            int64_t tbs, uint8_t* __restrict__ mapped, stormgpu_hit* h, int64_t* src) {
  const int lane = threadIdx.x & 31;
  const int P = pb.pcount[r];
  const int64_t s0 = pb.pstart[r];
  const bool rounds = pb.round_slots != nullptr;
  int lo = 0, hi = P, T = sp.min_score;
  if (rounds) {
    lo = pb.round_cur[2 * r];
    hi = pb.round_cur[2 * r + 1];
    if (pb.round > 0) T = pb.thr[r];
  }
  {
    bool loaded = false;
    for (int base = lo; base < hi; base += 32) {
      const int k = base + lane;
      const bool in = k < hi;
      const int score = in ? pb.a_score[s0 + k] : kMinScore;
      const int bound = in && score > T ? pb.a_bound[s0 + k] : kMinScore;
      unsigned m = __ballot_sync(0xffffffffu, in && score > T && bound >= T);
      if (m && !loaded) {
        loaded = true;
        const int32_t* g = reinterpret_cast<const int32_t*>(hits + r * 4);
        if (lane < 28) reinterpret_cast<int32_t*>(h)[lane] = g[lane];
        if (lane < 4) src[lane] = -1 - lane;
        __syncwarp();
      }
      while (m) {
        const int l = __ffs(m) - 1;
        const int sc = __shfl_sync(0xffffffffu, score, l);
        if (lane == 0) {
          hit_update(h, src, pb, sp, s0 + base + l, sc, ref_id, sense);
          if (h[3].score > T) T = h[3].score;
        }
        T = __shfl_sync(0xffffffffu, T, 0);
        m = __ballot_sync(0xffffffffu, in && lane > l && score > T && bound >= T);
      }
    }
    if (loaded) {
      __syncwarp();
      if (lane == 0) mapped[r] = 1;
      int32_t* g = reinterpret_cast<int32_t*>(hits + r * 4);
      if (lane < 28) g[lane] = reinterpret_cast<const int32_t*>(h)[lane];
      // rows in place only move to higher ranks: the highest rank first, every source is intact
      for (int q = 3; q >= 0; --q) {
        const int64_t f = src[q];
        if (f == -1 - q) continue;
        uint8_t* dst = tbo + (r * 4 + q) * tbs;
        if (f < 0) {
          const uint8_t* from = tbo + (r * 4 + (-1 - f)) * tbs;
          for (int64_t b = lane; b < tbs; b += 32) dst[b] = from[b];
        } else {
          const uint8_t* from = pb.a_tb + f * pb.tbs;
          const int tl = h[q].tb_len;
          for (int64_t b = lane; b < tbs; b += 32) {
            const int p = (int)(2 * b);
            int v = 0;
            if (p < tl) v = tbget(from, tl - 1 - p) << 4;
            if (p + 1 < tl) v |= tbget(from, tl - 2 - p);
            dst[b] = (uint8_t)v;
          }
        }
        __syncwarp();
      }
    }
  }
  if (!rounds) return;
  // the next round's candidates
  int end = hi, left = take;
  bool any = false;
  while (left > 0 && end < P) {
    const int k = end + lane;
    const bool in = k < P;
    const bool may = in && (!pb.ub || pb.ub[s0 + k] > T);
    unsigned m = __ballot_sync(0xffffffffu, may);
    int stop = min(32, P - end);
    if (__popc(m) >= left) {  // ends at the last one taken
      for (int over = __popc(m) - left; over > 0; --over) m &= ~(1u << (31 - __clz(m)));
      stop = 32 - __clz(m);
    }
    left -= __popc(m);
    any |= m != 0;
    unsigned long long b = 0;
    if (lane == 0 && m) b = atomicAdd(pb.round_count + 1, (unsigned long long)__popc(m));
    b = __shfl_sync(0xffffffffu, b, 0);
    if ((m >> lane) & 1u) pb.round_slots[b + __popc(m & ((1u << lane) - 1u))] = (int32_t)(s0 + k);
    else if (lane < stop) pb.a_score[s0 + k] = kMinScore;
    end += stop;
  }
  if (lane == 0 && any) {  // a read with no candidate left to select is done
    pb.round_cur[2 * r] = hi;
    pb.round_cur[2 * r + 1] = end;
    pb.thr[r] = T;
    pb.active_next[atomicAdd(pb.active_count + 1, 1)] = (int32_t)r;
  }
}

__global__ void __launch_bounds__(kReplayWarps * 32) replay_kernel(ScoreParams sp, int ref_id, int sense, PassBuffers pb,
                                                                   int take, stormgpu_hit* __restrict__ hits,
                                                                   uint8_t* __restrict__ tbo, int64_t tbs,
                                                                   uint8_t* __restrict__ mapped) {
  __shared__ stormgpu_hit sh_hits[kReplayWarps][4];
  __shared__ int64_t sh_src[kReplayWarps][4];
  const int w = threadIdx.x >> 5;
  const int n = *pb.active_count;
  for (int k = blockIdx.x * kReplayWarps + w; k < n; k += gridDim.x * kReplayWarps) {
    replay_read(pb.active[k], sp, ref_id, sense, pb, take, hits, tbo, tbs, mapped, sh_hits[w], sh_src[w]);
    __syncwarp();
  }
}

void launch_replay(int64_t n, const ScoreParams& sp, int ref_id, int sense, PassBuffers& pb, int take,
                   stormgpu_hit* hits, uint8_t* tb, int64_t tbs, uint8_t* mapped, cudaStream_t st) {
  if (n <= 0) return;
  const int64_t blocks = std::min<int64_t>((n + kReplayWarps - 1) / kReplayWarps,
                                           resident_grid(replay_kernel, kReplayWarps * 32));
  replay_kernel<<<(unsigned)blocks, kReplayWarps * 32, 0, st>>>(sp, ref_id, sense, pb, take, hits, tb, tbs, mapped);
}

// ------------------------------------------------------------------------------ slots of a read

__device__ __forceinline__ void slot_starts(int64_t npass, const int32_t* p_read, int32_t* pstart) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < npass; s += (int64_t)gridDim.x * blockDim.x) {
    const int r = p_read[s];
    if (s == 0 || p_read[s - 1] != r) pstart[r] = (int32_t)s;
  }
}

// Per read its number of slots, the list of reads with slots, and with rounds the first round's
// slots: the first `take` of each read (their bounds exceed -t, the threshold it starts from).  A
// slot's place in its read is the number of smaller diagonals of the read (they are distinct),
// counted here for reads with few slots; the others go to the long list.
__device__ __forceinline__ void slot_lists(int64_t npass, const KeptList& kl, int16_t* ub, const PassBuffers& pb, int take) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < npass; base += stride) {
    const int64_t s = base + lane;
    const bool in = s < npass;
    const int r = in ? pb.p_read[s] : -1;
    const int64_t s0 = in ? pb.pstart[r] : 0;
    const int rank = in ? (int)(s - s0) : -1;
    const bool last = in && (s == npass - 1 || pb.p_read[s + 1] != r);
    if (last) pb.pcount[r] = rank + 1;
    if (in) {
      const int32_t d = kl.diag[s];
      int smaller = 0, k = 0;
      for (; k <= kShortSlots && s0 + k < npass && pb.p_read[s0 + k] == r; ++k) smaller += kl.diag[s0 + k] < d;
      if (k <= kShortSlots) {
        pb.p_diag[s0 + smaller] = d;
        if (kl.ub) ub[s0 + smaller] = kl.ub[s];
      } else if (rank == 0) {
        kl.long_list[atomicAdd(kl.long_count, 1)] = r;
      }
    }
    const unsigned mf = __ballot_sync(0xffffffffu, rank == 0);
    if (mf) {
      int b = 0;
      if (lane == 0) b = atomicAdd(pb.active_count, __popc(mf));
      b = __shfl_sync(0xffffffffu, b, 0);
      if (rank == 0) pb.active[b + __popc(mf & ((1u << lane) - 1u))] = r;
    }
    if (!pb.round_slots) continue;
    const bool sel = in && rank < take;
    if (rank == 0) pb.round_cur[2 * r] = 0;
    if (sel && (last || rank == take - 1)) pb.round_cur[2 * r + 1] = rank + 1;
    const unsigned m = __ballot_sync(0xffffffffu, sel);
    if (m) {
      unsigned long long b = 0;
      if (lane == 0) b = atomicAdd(pb.round_count, (unsigned long long)__popc(m));
      b = __shfl_sync(0xffffffffu, b, 0);
      if (sel) pb.round_slots[b + __popc(m & ((1u << lane) - 1u))] = (int32_t)s;
    }
  }
}

// The reads of the long list, one warp each: their slots copied when they are ascending already (the
// block gather's reads), else sorted in shared memory as (diagonal, bound) keys.
constexpr int kSortWarps = 4;
__device__ __forceinline__ void slot_sort(const KeptList& kl, int16_t* ub, const PassBuffers& pb, int cap,
                                          unsigned long long* skeys) {  // cap per warp, a power of two
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long* a = skeys + (size_t)w * cap;
  const int n = *kl.long_count;
  for (int q = blockIdx.x * kSortWarps + w; q < n; q += gridDim.x * kSortWarps) {
    const int r = kl.long_list[q];
    const int P = pb.pcount[r];
    const int64_t s0 = pb.pstart[r];
    bool asc = true;
    for (int k = lane; k < P; k += 32) {
      const int32_t d = kl.diag[s0 + k];
      if (k > 0 && kl.diag[s0 + k - 1] > d) asc = false;
      pb.p_diag[s0 + k] = d;
      if (kl.ub) ub[s0 + k] = kl.ub[s0 + k];
    }
    if (__all_sync(0xffffffffu, asc) || P > cap) continue;  // a read above cap came from the block gather
    int N = 64;
    while (N < P) N <<= 1;
    for (int k = lane; k < N; k += 32)
      a[k] = k < P ? ((unsigned long long)((uint32_t)kl.diag[s0 + k] ^ 0x80000000u) << 32) |
                         (kl.ub ? (uint16_t)kl.ub[s0 + k] : 0u)
                   : ~0ull;
    __syncwarp();
    for (int k = 2; k <= N; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = lane; i < N; i += 32) {
          const int x = i ^ j;
          if (x > i) {
            const unsigned long long u = a[i], v = a[x];
            if ((u > v) == ((i & k) == 0)) { a[i] = v; a[x] = u; }
          }
        }
        __syncwarp();
      }
    for (int k = lane; k < P; k += 32) {
      pb.p_diag[s0 + k] = (int32_t)((uint32_t)(a[k] >> 32) ^ 0x80000000u);
      if (kl.ub) ub[s0 + k] = (int16_t)(uint16_t)a[k];
    }
    __syncwarp();
  }
}

__global__ void slot_starts_kernel(KeptList kl, PassBuffers pb) {
  slot_starts(kl.n_dev ? *kl.n_dev : kl.n, pb.p_read, pb.pstart);
}

__global__ void slot_lists_kernel(KeptList kl, int16_t* __restrict__ ub, PassBuffers pb, int take) {
  slot_lists(kl.n_dev ? *kl.n_dev : kl.n, kl, ub, pb, take);
}

__global__ void __launch_bounds__(kSortWarps * 32) slot_sort_kernel(KeptList kl, int16_t* __restrict__ ub, PassBuffers pb,
                                                                    int cap) {
  extern __shared__ unsigned long long skeys[];
  slot_sort(kl, ub, pb, cap, skeys);
}

// The three by one block, for a call of few reads (three launches of 2.5 to 5 us each).
__global__ void __launch_bounds__(kSortWarps * 32) slots_small_kernel(KeptList kl, int16_t* ub, PassBuffers pb, int take,
                                                                      int cap) {
  extern __shared__ unsigned long long skeys[];
  const int64_t n = kl.n_dev ? *kl.n_dev : kl.n;
  slot_starts(n, pb.p_read, pb.pstart);
  __syncthreads();
  slot_lists(n, kl, ub, pb, take);
  __syncthreads();
  slot_sort(kl, ub, pb, cap, skeys);
}

void launch_slot_lists(const KeptList& kl, int16_t* ub, PassBuffers& pb, int take, cudaStream_t st) {
  if (kl.n <= 0) return;
  int cap = 64;
  while (cap < kl.sort_cap) cap <<= 1;
  const size_t smem = (size_t)kSortWarps * cap * sizeof(unsigned long long);
  if (kl.n <= kSlotsSmall) {
    set_smem_attribute_once(reinterpret_cast<const void*>(slots_small_kernel), kSortWarps * 2048 * 8);
    slots_small_kernel<<<1, kSortWarps * 32, smem, st>>>(kl, ub, pb, take, cap);
    return;
  }
  const int64_t blocks = std::min<int64_t>((kl.n + 255) / 256, 148 * 32);
  slot_starts_kernel<<<(unsigned)blocks, 256, 0, st>>>(kl, pb);
  slot_lists_kernel<<<(unsigned)blocks, 256, 0, st>>>(kl, ub, pb, take);
  set_smem_attribute_once(reinterpret_cast<const void*>(slot_sort_kernel), kSortWarps * 2048 * 8);
  const int64_t grid = std::min<int64_t>((kl.n / kShortSlots + kSortWarps) / kSortWarps,
                                         resident_grid(slot_sort_kernel, kSortWarps * 32, smem));
  slot_sort_kernel<<<(unsigned)grid, kSortWarps * 32, smem, st>>>(kl, ub, pb, cap);
}

}  // namespace sg
