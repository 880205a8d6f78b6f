// map_kernels.cu -- the kernels of one mapping pass (one reference sequence x one strand).
//
//  (hit gather: gather.cu; banded filter: sw_filter.cu)
//  align                                            banded DP + traceback (alignment.c:488-734)
//  replay                                           per-read top-4 update (run.c:664-691,
//                                                   hit_map.c:50-144)
#include "map_kernels.cuh"

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

// Cell state packed in 16 bits: from (2) | indels (7) | colour checksum (2) | auto-correct (2)
// | freshness (3).  "from": 3 corner, 2 top, 1 left (alignment.c:13-19).
__device__ __forceinline__ int st_from(int s) { return s & 3; }
__device__ __forceinline__ int st_ind(int s) { return (s >> 2) & 127; }
__device__ __forceinline__ int st_chk(int s) { return (s >> 9) & 3; }
__device__ __forceinline__ int st_ac(int s) { return (s >> 11) & 3; }
__device__ __forceinline__ int st_fr(int s) { return (s >> 13) & 7; }
__device__ __forceinline__ int st_make(int from, int ind, int chk, int ac, int fr) {
  return from | (ind << 2) | (chk << 9) | (ac << 11) | (fr << 13);
}

constexpr int kMaxBand = 2 * STORMGPU_MAX_INDELS + 1;

// The colour state of a corner step (alignment.c:535-603, and the condition of the SNP adjustment
// :465-468) as a table: index = state of the corner cell (checksum | auto-correct << 2 | freshness << 4)
// | checksum of the cell's own colours << 7 | quality level << 9; entry = the new state, bit 7 the
// condition.  The branches of the state machine, taken differently in every lane, were most of the
// colour alignment's time (one round of 300 reads of 49 colours, both strands: 0.58 -> 0.31 ms).
constexpr int kColourTable = 2048;
__device__ __forceinline__ uint8_t colour_step(int idx) {
  const int cchk = idx & 3, cac = (idx >> 2) & 3, cfr = (idx >> 4) & 7, chk0 = (idx >> 7) & 3, q = (idx >> 9) & 3;
  int chk = chk0 ^ cchk, ac = chk0, fr = chk0 ? q : 0;
  if (cchk != chk) {
    if (cchk == 0) { ac = chk; fr = q; }
    else if (chk == cac) { ac = 0; chk = 0; fr = 0; }
    else if (chk == 0) { if (cfr - 1 > 0) { ac = cac; fr = cfr - 1; } else { ac = 0; fr = 0; } }
    else { if (cfr - 1 > 0) { ac = cac; fr = cfr - 1; } else { ac = chk; fr = q; } }
  } else {
    if (cac != 0) {
      if (cfr - 1 > 0) {
        if (chk == 0) { ac = 0; fr = 0; } else { ac = cac; fr = cfr - 1; }
      }
    } else { chk = 0; ac = 0; fr = 0; }
  }
  const int cmp = cchk ^ chk0;
  const bool adjust = cchk && (cmp == 0 || cmp == cac);
  return (uint8_t)(chk | (ac << 2) | (fr << 4) | (adjust ? 0x80 : 0));
}

// alignment.c:326-360 (init), :488-632 (rows 1..L-1, corner > top > left on ties, gaps only
// while indels < I, affine through the predecessor's direction, colour checksum state
// machine :535-603 with the SNP adjustment :465-468), best cell on the last row (:621-630),
// traceback :642-734.  The direction of every cell (2 bits) and, in colour space, whether its
// pair score was made positive by the SNP adjustment (the `score > corner score` test of
// :693) go to the scratch, column-minor: word (row*wpr + k)*ns + sl for scratch column sl of
// ns (the slot's index in a one-per-thread launch, the thread's index in a persistent one).
// Genome and mask codes of the band of one row, 2 bits each in registers, for a constant band
// width: row i + 1 is row i moved by one code, so each row loads one genome and one mask code
// (instead of BW of each).
template <int BWT>
struct BandWindow {
  static_assert(BWT > 0 && BWT <= 64, "band width");
  uint64_t g[2] = {0, 0}, m[2] = {0, 0};
  __device__ __forceinline__ void put(int c, int gc, int mc) {
    g[c >> 5] |= (uint64_t)gc << (2 * (c & 31));
    m[c >> 5] |= (uint64_t)mc << (2 * (c & 31));
  }
  // codes [base, base + BWT)
  __device__ __forceinline__ void load(const uint8_t* genome, const uint8_t* mask, int64_t base) {
#pragma unroll
    for (int c = 0; c < BWT; ++c) put(c, code_at(genome, base + c), code_at(mask, base + c));
  }
  // drop cell 0, the others move down one cell, code `pos` becomes cell BWT - 1
  __device__ __forceinline__ void advance(const uint8_t* genome, const uint8_t* mask, int64_t pos) {
    if (BWT > 32) {
      g[0] = (g[0] >> 2) | (g[1] << 62);
      m[0] = (m[0] >> 2) | (m[1] << 62);
      g[1] >>= 2;
      m[1] >>= 2;
    } else {
      g[0] >>= 2;
      m[0] >>= 2;
    }
    put(BWT - 1, code_at(genome, pos), code_at(mask, pos));
  }
  __device__ __forceinline__ int gcode(int c) const { return (int)((g[c >> 5] >> (2 * (c & 31))) & 3u); }
  __device__ __forceinline__ int mcode(int c) const { return (int)((m[c >> 5] >> (2 * (c & 31))) & 3u); }
};

// Traceback over the direction words of the rows from i (cell c) up: emit(i, c, words of the row,
// direction) for every cell of the path.  A path leaves a row once (every step but LEFT goes up), so the
// rows' words are loaded four rows ahead whatever the path does; walked one cell at a time, each
// step waited for its own word.
template <int WPR, int WDIR, int LEFT, int TOP, class Emit>
__device__ __forceinline__ void trace_rows(const uint32_t* scr, int64_t ns, int64_t sl, int i, int c, int BW, Emit emit) {
  constexpr int PF = 4;
  uint32_t w[PF][WPR];
  auto load = [&](int q, int row) {
#pragma unroll
    for (int k = 0; k < WPR; ++k) w[q][k] = row >= 0 ? scr[((int64_t)row * WPR + k) * ns + sl] : 0u;
  };
#pragma unroll
  for (int q = 0; q < PF; ++q) load(q, i - q);
  for (;;) {
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      int from;
      for (;;) {
        uint32_t x = w[q][0];
        if (WDIR > 1 && c >= 16) x = w[q][WDIR > 1 ? 1 : 0];
        if (WDIR > 2 && c >= 32) x = w[q][WDIR > 2 ? 2 : 0];
        from = (x >> ((2 * c) & 31)) & 3;
        emit(i, c, w[q], from);
        if (from != LEFT) break;
        if (--c < 0) return;
      }
      if (from == TOP) ++c;
      if (--i < 0 || c >= BW) return;
      load(q, i - (PF - 1));
    }
  }
}

// BWT > 0: the band width 2I + 1 as a constant, so that the row arrays live in registers;
// BWT = 0: any width up to kMaxBand (arrays in local memory).  ctab: the table of colour_step.  CM: 0 nucleotide, 1 colour
// space (the colour state machine compiled in), -1 either (sp.colour); the kernel's CM = 2 runs
// the packed nucleotide form below (align_one_nuc).
// A candidate whose running abort bound falls below the replay's threshold stops at that row:
// -t, or with rounds the running threshold its read had after the rounds before (the replay's
// threshold only rises, so the candidate is aborted whatever comes before it), and neither its
// score nor its traceback is read.
// One slot; its direction bits in scratch column sl of ns.  Returns the rows it computed.
template <int BWT, int CM>
__device__ __forceinline__ int align_one(const ReadsDev& rd, const ScoreParams& sp, const uint8_t* __restrict__ genome,
                                         const uint8_t* __restrict__ mask, int64_t slot, int64_t sl, int64_t ns,
                                         const PassBuffers& pb, const uint8_t* ctab) {
  constexpr int NB = BWT > 0 ? BWT : kMaxBand;
  const int r = pb.p_read[slot];
  // the first round, and a launch without rounds, stop at -t only: pb.thr holds the read's
  // threshold after the rounds before this one (in the first round, a previous pass's value)
  const int thr = (pb.thr && pb.round > 0) ? max(sp.min_score, pb.thr[r]) : sp.min_score;
  const int d = pb.p_diag[slot];
  const int I = sp.I, BW = BWT > 0 ? BWT : 2 * I + 1, colour = CM >= 0 ? CM : sp.colour;
  const int L = rd.lengths[r];
  const uint8_t* rdc = rd.codes + (int64_t)r * rd.cstride;
  const uint8_t* rdq = rd.levels ? rd.levels + (int64_t)r * rd.lstride : nullptr;
  const int win = max(d - I, -sp.Is);  // run.c:667
  const int wpr_dir = (2 * BW + 31) / 32, wpr = wpr_dir + (colour ? (BW + 31) / 32 : 0);
  uint32_t* scr = pb.a_scratch;
  int sc[NB], stt[NB];
  const int mbest = sp.pair[0][3];
  BandWindow<(BWT > 0 ? BWT : 1)> bwin;
  if (BWT > 0) bwin.load(genome, mask, win);
  // row 0
  {
    const int rc = code_at(rdc, 0), q = rdq ? code_at(rdq, 0) : 3;
    uint32_t wd[(2 * NB + 31) / 32] = {};
#pragma unroll
    for (int c = 0; c < BW; ++c) {
      const int64_t j = (int64_t)win + c;
      const int f = BWT > 0 ? bwin.gcode(c) : code_at(genome, j);
      int chk = 0, score;
      if ((BWT > 0 ? bwin.mcode(c) : code_at(mask, j)) == 0) {
        chk = colour ? (rc ^ f) : 0;
        score = sp.pair[colour ? (chk ? 1 : 0) : (rc != f)][q];
      } else score = kMinScore;
      sc[c] = score;
      stt[c] = st_make(3, 0, chk, chk, (colour && chk) ? q : 0);
      wd[(2 * c) >> 5] |= 3u << ((2 * c) & 31);
    }
    for (int k = 0; k < wpr; ++k) scr[(int64_t)k * ns + sl] = k < wpr_dir ? wd[k] : 0u;
  }
  int best_possible = (colour ? (L - 2) : L) * mbest;
  long long bound = 0x7fffffffLL;
  int rows = L;
  for (int i = 1; i < L; ++i) {
    const int rc = code_at(rdc, i), q = rdq ? code_at(rdq, i) : 3;
    int max_on_line = kMinScore;
    int lsc = kMinScore, lst = st_make(3, I, 0, 0, 0);  // left border
    uint32_t wd[(2 * NB + 31) / 32] = {};
    uint32_t wc[(NB + 31) / 32] = {};
    if (BWT > 0) bwin.advance(genome, mask, (int64_t)win + i + BW - 1);
#pragma unroll
    for (int c = 0; c < BW; ++c) {
      const int64_t j = (int64_t)win + i + c;
      const int f = BWT > 0 ? bwin.gcode(c) : code_at(genome, j);
      // initial values of this cell (alignment__init_matrix)
      int chk0 = 0, ac0 = 0, fr0 = 0, s0;
      if ((BWT > 0 ? bwin.mcode(c) : code_at(mask, j)) == 0) {
        if (colour) { chk0 = ac0 = rc ^ f; fr0 = ac0 ? q : 0; s0 = sp.pair[chk0 ? 1 : 0][q]; }
        else s0 = sp.pair[rc != f][q];
      } else s0 = kMinScore;
      const int csc = sc[c], cst = stt[c];
      const int tsc = c + 1 < BW ? sc[c + 1] : kMinScore;
      const int tst = c + 1 < BW ? stt[c + 1] : st_make(3, I, 0, 0, 0);
      int ms = s0, step = 0;
      if (colour) {
        step = ctab[(cst >> 9) | (chk0 << 7) | (q << 9)];
        if ((step & 0x80) && s0 != kMinScore && s0 < 0) ms = -2 * s0;
      }
      int score = csc + ms, it = 0, tmp;
      if (st_ind(tst) < I && (tmp = tsc + ((st_from(tst) ^ 2) ? sp.gap_open : sp.gap_ext)) > score) { it = 1; score = tmp; }
      if (st_ind(lst) < I && (tmp = lsc + ((st_from(lst) ^ 1) ? sp.gap_open : sp.gap_ext)) > score) { it = 2; score = tmp; }
      // the state after a corner, or after a gap: one more indel, the gap's own checksum, and the
      // source's freshness less one while it lasts
      const int gst = it == 1 ? tst : lst;
      int nst;
      if (colour) {
        const bool fresh = st_fr(gst) > 1;
        const int gap = st_make(it == 1 ? 2 : 1, st_ind(gst) + 1, st_chk(gst) ^ (it == 1 ? rc : f),
                                fresh ? st_ac(cst) : ac0, fresh ? st_fr(gst) - 1 : fr0);
        nst = it == 0 ? (3 | (cst & 0x1FC) | ((step & 0x7F) << 9)) : gap;
      } else {
        nst = it == 0 ? (3 | (cst & 0x1FC)) : (3 - it) | ((st_ind(gst) + 1) << 2);
      }
      const int from = nst & 3;
      sc[c] = score;
      stt[c] = nst;
      lsc = score;
      lst = nst;
      if (max_on_line < score) max_on_line = score;
      wd[(2 * c) >> 5] |= (uint32_t)from << ((2 * c) & 31);
      if (colour && it == 0 && ms > 0) wc[c >> 5] |= 1u << (c & 31);
    }
    if ((long long)max_on_line + best_possible < bound) bound = (long long)max_on_line + best_possible;
    best_possible -= mbest;
    for (int k = 0; k < wpr_dir; ++k) scr[((int64_t)i * wpr + k) * ns + sl] = wd[k];
    if (colour)
      for (int k = wpr_dir; k < wpr; ++k) scr[((int64_t)i * wpr + k) * ns + sl] = wc[k - wpr_dir];
    if (bound < thr) {  // aborted at any threshold it can meet
      rows = i + 1;
      break;
    }
  }
  int best = kMinScore, bi = -1, bj = -1;
#pragma unroll
  for (int c = 0; c < BW; ++c)
    if (best < sc[c]) { best = sc[c]; bi = L - 1; bj = L - 1 + c; }
  const int32_t bnd = bound > 0x7fffffffLL ? 0x7fffffff : (int32_t)bound;
  pb.a_score[slot] = best;
  pb.a_bound[slot] = bnd;
  int i0 = bi, j0 = bj, tl = 0;
  uint8_t* tb = pb.a_tb + slot * pb.tbs;
  if (bi >= 0 && bnd >= thr && best > thr) {
    int colr = 0;
    uint8_t cur = 0;
    auto put = [&](int op) {
      if (tl & 1) { cur |= (uint8_t)op; tb[tl >> 1] = cur; }
      else { cur = (uint8_t)(op << 4); tb[tl >> 1] = cur; }
      tl++;
    };
    // one cell: its operation; adj: its pair score was made positive by the SNP adjustment
    auto cell = [&](int i, int c, int from, bool adj) {
      const int j = i + c;
      i0 = i;
      j0 = j;
      const int rc = code_at(rdc, i);
      if (from == 2) { put(0xC | rc); return; }
      if (from == 1) { put(0x1); return; }
      const int f = code_at(genome, (int64_t)win + j);
      if (rc == f) put(0x3);
      else if (!colour || !(colr || (adj && i != 0 && j != 0))) put(0x4 | rc);
      else { put(0x8 | rc); colr ^= rc ^ f; }
    };
    if constexpr (BWT > 0) {
      constexpr int WD = (2 * BWT + 31) / 32, WC = CM == 0 ? 0 : (BWT + 31) / 32;
      trace_rows<WD + WC, WD, 1, 2>(scr, ns, sl, bi, bj - bi, BW, [&](int i, int c, const uint32_t* w, int from) {
        uint32_t x = 0;
        if (WC > 0) x = w[WC > 0 ? WD : 0];
        if (WC > 1 && c >= 32) x = w[WC > 1 ? WD + 1 : 0];
        cell(i, c, from, WC > 0 && ((x >> (c & 31)) & 1u));
      });
    } else {
      int i = bi, c = bj - bi;
      while (i >= 0 && i < L && c >= 0 && c < BW) {
        const uint32_t wdir = scr[((int64_t)i * wpr + ((2 * c) >> 5)) * ns + sl];
        const int from = (wdir >> ((2 * c) & 31)) & 3;
        const bool adj = colour && ((scr[((int64_t)i * wpr + wpr_dir + (c >> 5)) * ns + sl] >> (c & 31)) & 1u);
        cell(i, c, from, adj);
        if (from == 2) { i--; c++; }
        else if (from == 1) { c--; }
        else { i--; }
      }
    }
  }
  pb.a_tblen[slot] = tl;
  pb.a_pos[slot * 4 + 0] = (int16_t)bi;
  pb.a_pos[slot * 4 + 1] = (int16_t)bj;
  pb.a_pos[slot * 4 + 2] = (int16_t)i0;
  pb.a_pos[slot * 4 + 3] = (int16_t)j0;
  return rows;
}

// Nucleotide space with a constant band: the DP of align_one with each cell in one register,
//   score << 13 | from << 10 (one-hot: corner 4, top 2, left 1) | guard << 8 | ind',
// ind' = indels + 256 - I in 8 bits, whose carry into the guard bit marks indels == I (no gap
// may leave such a cell).  The largest candidate value is the reference's choice
// (alignment.c:521-532: the higher score, on equal scores corner before top before left) and
// carries its direction and indel count, so a cell is one three-way max.  The gap candidates
// are formed with integer multiply-adds, which issue on the FMA pipe beside the ALU's logic and
// max operations: t + (open << 13 | 1) relabelled as a gap, plus (t & (its from bit | guard))
// times a constant K chosen modulo 2^32 so that the from bit adds (ext - open) << 13 (an
// extension) and the guard about -2^30, which puts a gap the reference does not allow below
// every cell.  Direction bits are moved into the row's words by multiply-adds too.
// Cells are floored at score -2^16 (every 16 rows, and in rows with masked cells): a floored
// cell, and any cell whose value derives from one, stays below -2^16 + L * (largest pair score),
// under the row maximum's start MIN_SCORE and below every cell of a path the replay can keep
// (sp.packed holds only when -t - L * match stays above it); so every score, bound and traceback
// the replay reads is the reference's, and no packed value overflows.
constexpr int kCellShift = 13;
constexpr int kCellFloor = -(1 << 29);
constexpr uint32_t kFromC = 1u << 12, kFromT = 1u << 11, kFromL = 1u << 10, kFromAll = kFromC | kFromT | kFromL;
constexpr uint32_t kGuard = 1u << 8;

__device__ __forceinline__ uint32_t mad_lo(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t mad_hi(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// One row of the packed DP: v[] holds the previous row and becomes this one; mis / msk hold a
// bit at 2c for a mismatching / masked cell c (word c >> 4); returns the row maximum.  The
// corner relabelling of v[c + 1] serves both this cell's top candidate and the next cell's
// corner.  Rows without masked cells skip the floor (align_one_nuc floors every cell every 16
// rows: between those a cell falls by at most 16 * 255 << 13, so nothing overflows and a gap
// the reference forbids still lands below every cell); rows with masked cells (MIN_SCORE)
// floor every cell.
template <int BW, bool MASKED>
__device__ __forceinline__ int packed_row(int (&v)[BW], uint32_t (&wd)[(2 * BW + 31) / 32], const uint32_t* mis,
                                          const uint32_t* msk, int SM, int SX, int MINS, const ScoreParams& sp) {
  int mol = MINS, left = 0, pend = MINS;
  uint32_t cv = ((uint32_t)v[0] & ~kFromAll) | kFromC;  // v[c] relabelled as a corner source
#pragma unroll
  for (int c = 0; c < BW; ++c) {
    const uint32_t bit = 1u << (2 * (c & 15));
    int s0 = (mis[c >> 4] & bit) ? SX : SM;
    if (MASKED && (msk[c >> 4] & bit)) s0 = MINS;
    int nv = (int)mad_lo((uint32_t)s0, sp.one, cv);
    if (MASKED) nv = max(nv, kCellFloor);
    int top = 0, lft = 0;
    if (c + 1 < BW) {
      const uint32_t t = (uint32_t)v[c + 1];
      cv = (t & ~kFromAll) | kFromC;
      top = (int)mad_lo(t & (kFromT | kGuard), sp.kt, mad_lo(cv, sp.one, sp.open1_tc));
    }
    if (c > 0) {
      const uint32_t l = (uint32_t)left;
      const uint32_t b = (mad_lo(l, sp.one, sp.open1) & ~kFromAll) | kFromL;
      lft = (int)mad_lo(l & (kFromL | kGuard), sp.kl, b);
    }
    if (c > 0 && c + 1 < BW) nv = __vimax3_s32(nv, top, lft);
    else if (c + 1 < BW) nv = max(nv, top);
    else if (c > 0) nv = max(nv, lft);
    v[c] = nv;
    left = nv;
    if (c & 1) mol = __vimax3_s32(mol, pend, nv);
    else if (c + 1 == BW) mol = max(mol, nv);
    else pend = nv;
    const uint32_t x = (uint32_t)nv & (kFromC | kFromT);  // direction: 2 corner, 1 top, 0 left
    const int p = 2 * (c & 15);
    if (p <= 10) wd[c >> 4] = mad_hi(x, sp.pw[21 + p], wd[c >> 4]);
    else wd[c >> 4] = mad_lo(x, sp.pw[p - 11], wd[c >> 4]);
  }
  return mol;
}

template <int BW>
__device__ __forceinline__ int align_one_nuc(const ReadsDev& rd, const ScoreParams& sp,
                                             const uint8_t* __restrict__ genome, const uint8_t* __restrict__ mask,
                                             int64_t slot, int64_t sl, int64_t ns, const PassBuffers& pb) {
  static_assert(BW <= 48, "three direction words per row at most");
  const int r = pb.p_read[slot];
  const int thr = (pb.thr && pb.round > 0) ? max(sp.min_score, pb.thr[r]) : sp.min_score;
  const int d = pb.p_diag[slot];
  const int I = sp.I;
  const int L = rd.lengths[r];
  const uint8_t* rdc = rd.codes + (int64_t)r * rd.cstride;
  const uint8_t* rdq = rd.levels ? rd.levels + (int64_t)r * rd.lstride : nullptr;
  const int win = max(d - I, -sp.Is);  // run.c:667
  constexpr int wpr = (2 * BW + 31) / 32;
  constexpr int NW64 = (BW + 31) / 32;
  uint32_t* scr = pb.a_scratch;
  const int MINS = kMinScore * (1 << kCellShift);
  int v[BW];
  const int mbest = sp.pair[0][3];
  BandWindow<BW> bwin;
  bwin.load(genome, mask, win);
  {  // row 0: pair scores only (alignment.c:326-360); indels 0
    const int rc = code_at(rdc, 0), q = rdq ? code_at(rdq, 0) : 3;
    const int SM = sp.pair[0][q] * (1 << kCellShift), SX = sp.pair[1][q] * (1 << kCellShift);
    const int init = (int)kFromC | (256 - I);
    uint32_t wd[wpr] = {};
#pragma unroll
    for (int c = 0; c < BW; ++c) {
      v[c] = (bwin.mcode(c) == 0 ? (rc != bwin.gcode(c) ? SX : SM) : MINS) | init;
      wd[(2 * c) >> 5] |= 2u << ((2 * c) & 31);
    }
#pragma unroll
    for (int k = 0; k < wpr; ++k) scr[(int64_t)k * ns + sl] = wd[k];
  }
  int best_possible = L * mbest;
  long long bound = 0x7fffffffLL;
  int rows = L;
  for (int i = 1; i < L; ++i) {
    const int rc = code_at(rdc, i), q = rdq ? code_at(rdq, i) : 3;
    const int SM = sp.pair[0][q] * (1 << kCellShift), SX = sp.pair[1][q] * (1 << kCellShift);
    bwin.advance(genome, mask, (int64_t)win + i + BW - 1);
    uint32_t mis[2 * NW64], msk[2 * NW64];
    bool masked = false;
    const uint64_t rrep = (uint64_t)rc * 0x5555555555555555ull;
#pragma unroll
    for (int k = 0; k < NW64; ++k) {
      const uint64_t x = bwin.g[k] ^ rrep;
      const uint64_t mm = (x | (x >> 1)) & 0x5555555555555555ull;
      const uint64_t mk = (bwin.m[k] | (bwin.m[k] >> 1)) & 0x5555555555555555ull;
      mis[2 * k] = (uint32_t)mm;
      mis[2 * k + 1] = (uint32_t)(mm >> 32);
      msk[2 * k] = (uint32_t)mk;
      msk[2 * k + 1] = (uint32_t)(mk >> 32);
      masked |= mk != 0;
    }
    uint32_t wd[wpr] = {};
    if ((i & 15) == 0) {
#pragma unroll
      for (int c = 0; c < BW; ++c) v[c] = max(v[c], kCellFloor);
    }
    const int mol = masked ? packed_row<BW, true>(v, wd, mis, msk, SM, SX, MINS, sp)
                           : packed_row<BW, false>(v, wd, mis, msk, SM, SX, MINS, sp);
    const long long ml = (long long)(mol >> kCellShift) + best_possible;
    if (ml < bound) bound = ml;
    best_possible -= mbest;
#pragma unroll
    for (int k = 0; k < wpr; ++k) scr[((int64_t)i * wpr + k) * ns + sl] = wd[k];
    if (bound < thr) {
      rows = i + 1;
      break;
    }
  }
  int best = kMinScore, bi = -1, bj = -1;
#pragma unroll
  for (int c = 0; c < BW; ++c) {
    const int s = v[c] >> kCellShift;
    if (best < s) { best = s; bi = L - 1; bj = L - 1 + c; }
  }
  const int32_t bnd = bound > 0x7fffffffLL ? 0x7fffffff : (int32_t)bound;
  pb.a_score[slot] = best;
  pb.a_bound[slot] = bnd;
  int i0 = bi, j0 = bj, tl = 0;
  uint8_t* tb = pb.a_tb + slot * pb.tbs;
  if (bi >= 0 && bnd >= thr && best > thr) {  // alignment.c:642-734
    uint8_t cur = 0;
    // directions: 2 corner, 1 top, 0 left
    trace_rows<wpr, wpr, 0, 1>(scr, ns, sl, bi, bj - bi, BW, [&](int i, int c, const uint32_t*, int from) {
      const int j = i + c;
      i0 = i;
      j0 = j;
      const int rc = code_at(rdc, i);
      int op;
      if (from == 1) op = 0xC | rc;
      else if (from == 0) op = 0x1;
      else op = rc != code_at(genome, (int64_t)win + j) ? 0x4 | rc : 0x3;
      if (tl & 1) { cur |= (uint8_t)op; tb[tl >> 1] = cur; }
      else { cur = (uint8_t)(op << 4); tb[tl >> 1] = cur; }
      tl++;
    });
  }
  pb.a_tblen[slot] = tl;
  pb.a_pos[slot * 4 + 0] = (int16_t)bi;
  pb.a_pos[slot * 4 + 1] = (int16_t)bj;
  pb.a_pos[slot * 4 + 2] = (int16_t)i0;
  pb.a_pos[slot * 4 + 3] = (int16_t)j0;
  return rows;
}

// Slots slot0 .. slot0 + nslots: one per thread (scratch column = slot - slot0), or with
// pb.cursor a persistent grid whose warps take the next 32 slots from the cursor (the slot
// count read from pb.npass_dev when it is given; scratch column = the thread's index in the
// grid, so the scratch holds align_workers() columns).
// whether any code of [a, b) is masked
__device__ __forceinline__ bool window_masked(const uint8_t* __restrict__ mask, int64_t a, int64_t b) {
  unsigned any = 0;
  for (int64_t k = a >> 2; k <= (b - 1) >> 2; ++k) {
    unsigned x = mask[k];
    if (k == a >> 2) x &= 0xFFu << (2 * (a & 3));
    if (k == (b - 1) >> 2) x &= 0xFFu >> (6 - 2 * ((b - 1) & 3));
    any |= x;
  }
  return any != 0;
}

// Resident blocks of 128 threads per SM the registers are bounded for: the packed form holds about
// BWT registers of cells, the general one (scores and states apart) twice that.
constexpr int align_blocks(int bw, int cm) {
  return bw <= 0 ? 1 : cm == 3 ? 2 : cm == 2 ? (bw <= 15 ? 7 : bw <= 23 ? 6 : bw <= 31 ? 5 : 4) : (bw <= 15 ? 5 : bw <= 31 ? 4 : 3);
}

template <int BWT, int CM>
__global__ void __launch_bounds__(128, align_blocks(BWT, CM)) align_kernel(ReadsDev rd, ScoreParams sp,
                                                    const uint8_t* __restrict__ genome,
                                                    const uint8_t* __restrict__ mask, int64_t slot0, int64_t nslots,
                                                    PassBuffers pb) {
  __shared__ uint8_t ctab[CM == 1 || CM == -1 ? kColourTable : 1];
  if (CM == 1 || CM == -1) {
    for (int k = threadIdx.x; k < kColourTable; k += blockDim.x) ctab[k] = colour_step(k);
    __syncthreads();
  }
  // one call site of align_one (its band code is large and fully unrolled)
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool steal = pb.cursor != nullptr;
  int64_t n = steal && pb.npass_dev ? *pb.npass_dev : nslots;
  if (pb.round_slots) n = (int64_t)*pb.round_count;  // with rounds: round_slots[0 .. n)
  if (n <= pb.wave) return;                          // align_wave_kernel's
  const int64_t ns = steal ? (int64_t)gridDim.x * blockDim.x : nslots;
  const int lane = threadIdx.x & 31;
  const int take = pb.steal >= 32 ? pb.steal & ~31 : 32;
  unsigned long long rows = 0;
  int64_t s = tid, end = steal ? 0 : tid + 1;  // stealing: every lane takes the first run together
  for (;;) {
    if (steal && s >= end) {  // the warp's next run of `take` slots
      unsigned long long b = 0;
      if (lane == 0) b = atomicAdd(pb.cursor, (unsigned long long)take);
      s = (int64_t)__shfl_sync(0xffffffffu, b, 0);
      if (s >= n) break;
      end = s + take;
      s += lane;
    }
    if (s < n) {
      const int64_t slot = pb.round_slots ? (int64_t)pb.round_slots[s] : slot0 + s;
      if constexpr (CM == 2) {
        rows += (unsigned long long)align_one_nuc<BWT>(rd, sp, genome, mask, slot, steal ? tid : s, ns, pb);
      } else if constexpr (CM == 3) {
        // every cell exact: without masked codes no cell comes near the packed form's floor
        const int r = pb.p_read[slot];
        const int64_t win = max(pb.p_diag[slot] - sp.I, -sp.Is);
        if (window_masked(mask, win, win + rd.lengths[r] + 2 * sp.I))
          rows += (unsigned long long)align_one<BWT, 0>(rd, sp, genome, mask, slot, steal ? tid : s, ns, pb, ctab);
        else
          rows += (unsigned long long)align_one_nuc<BWT>(rd, sp, genome, mask, slot, steal ? tid : s, ns, pb);
      } else {
        rows += (unsigned long long)align_one<BWT, CM>(rd, sp, genome, mask, slot, steal ? tid : s, ns, pb, ctab);
      }
    }
    if (!steal) break;
    s += 32;
  }
  if (pb.cells) {
    for (int o = 16; o > 0; o >>= 1) rows += __shfl_xor_sync(0xffffffffu, rows, o);
    if (lane == 0 && rows) atomicAdd(pb.cells, rows * (unsigned long long)(2 * sp.I + 1));
  }
}

// The packed nucleotide form has every band width up to 41 as a constant (the general form in local
// memory ran -i 5 at 50 GCUPS, a twentieth of the packed form's rate); the others the widths of the
// filter's own limits and of -i 20.
static const void* align_kernel_of(const ScoreParams& sp) {
  if (sp.packed == 2) {
#define SG_ALIGN(BW) case BW: return (const void*)align_kernel<BW, 3>;
    switch (2 * sp.I + 1) { SG_ALIGN(7) SG_ALIGN(11) SG_ALIGN(15) SG_ALIGN(21) SG_ALIGN(31) SG_ALIGN(41) }
#undef SG_ALIGN
  } else if (sp.packed) {
#define SG_ALIGN(BW) case BW: return (const void*)align_kernel<BW, 2>;
    switch (2 * sp.I + 1) {
      SG_ALIGN(3) SG_ALIGN(5) SG_ALIGN(7) SG_ALIGN(9) SG_ALIGN(11) SG_ALIGN(13) SG_ALIGN(15) SG_ALIGN(17)
      SG_ALIGN(19) SG_ALIGN(21) SG_ALIGN(23) SG_ALIGN(25) SG_ALIGN(27) SG_ALIGN(29) SG_ALIGN(31) SG_ALIGN(33)
      SG_ALIGN(35) SG_ALIGN(37) SG_ALIGN(39) SG_ALIGN(41)
    }
#undef SG_ALIGN
  }
#define SG_ALIGN(BW) \
  case BW: return sp.colour ? (const void*)align_kernel<BW, 1> : (const void*)align_kernel<BW, 0>;
  switch (2 * sp.I + 1) {
    SG_ALIGN(7)
    SG_ALIGN(11)
    SG_ALIGN(15)
    SG_ALIGN(31)
    SG_ALIGN(41)
  default: return (const void*)align_kernel<0, -1>;
  }
#undef SG_ALIGN
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
// 800 windows of 101 codes take 75 us at -i 15 where a thread each takes 148, 88 us in colours at -i 7
// against 260 (the whole call).  The chain of a step (shuffle, sums, state, next row's codes) is what
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
