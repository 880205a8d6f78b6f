// align_core.cuh -- the banded full alignment with traceback (alignment.c:488-734), one candidate per
// thread: the kernel template and its forms.  They are instantiated in translation units of their own
// (align_packed.cu, align_unit.cu, align_general.cu), as the filter's and the score bound's are: the first
// use of a kernel loads its whole module, about 0.35 ms per MB, so that every form's code in one module cost
// the first mapping call of a process 4 ms (16 reads: 7.9 ms, 3.6 with the modules apart).
#pragma once

#include "map_kernels.cuh"

namespace sg {

// The instantiated kernels by band width (null: none for it).
const void* align_packed_kernel(int bw);              // CM 2: nucleotides, every odd width from 3 to 41
const void* align_unit_kernel(int bw);                // CM 3: the unit entry points
const void* align_general_kernel(int bw, int colour); // CM 0, 1; any width

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

// Traceback over the direction words of the rows from i (cell c) up: emit(i, c, direction) for every cell of
// the path.  A path leaves a row once (every step but LEFT goes up), so the rows' words are loaded four rows
// ahead whatever the path does; walked one cell at a time, each step waits for its own word.  For the
// candidates that a mapping aligns, whose paths are long and have few gaps: 9,001 reads of up to 251 codes at
// -i 5, alignments 4.95 ms, 5.18 without (12,000 of 100 codes at -i 20: 17.3 and 16.8).  In windows whose paths wander, as the unit entry points get them, the
// lanes of a warp part in it, and every form is faster without (see align_one).
template <int WPR, int LEFT, int TOP, class Emit>
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
        if (WPR > 1 && c >= 16) x = w[q][WPR > 1 ? 1 : 0];
        if (WPR > 2 && c >= 32) x = w[q][WPR > 2 ? 2 : 0];
        from = (x >> ((2 * c) & 31)) & 3;
        emit(i, c, from);
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
// BWT = 0: any width up to kMaxBand (arrays in local memory).  CM: 0 nucleotide, 1 colour space (the
// colour state machine compiled in; ctab: the table of colour_step); the kernel's CM = 2 and 3 run the
// packed nucleotide form below (align_one_nuc).  (With the space a run-time value the widths without a
// constant ran at less than half the rate in nucleotides: one window at -i 16 1.05 ms, now 0.43.)
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
  const int I = sp.I, BW = BWT > 0 ? BWT : 2 * I + 1, colour = CM;
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
    // (with the direction words loaded rows ahead as in trace_rows: 10,000 windows at -i 15 464 us, without 231;
    // 5,000 of 101 colours at -i 7 445 and 300)
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

template <int BW, bool AHEAD>
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
    auto cell = [&](int i, int c, int from) {
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
    };
    if (AHEAD) {
      trace_rows<wpr, 0, 1>(scr, ns, sl, bi, bj - bi, BW, cell);
    } else {
      int i = bi, c = bj - bi;
      while (i >= 0 && i < L && c >= 0 && c < BW) {
        const uint32_t wdir = scr[((int64_t)i * wpr + ((2 * c) >> 5)) * ns + sl];
        const int from = (wdir >> ((2 * c) & 31)) & 3;
        cell(i, c, from);
        if (from == 1) { i--; c++; }
        else if (from == 0) { c--; }
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

// Slots slot0 .. slot0 + nslots: one per thread (scratch column = slot - slot0), or with
// pb.cursor a persistent grid whose warps take the next 32 slots from the cursor (the slot
// count read from pb.npass_dev when it is given; scratch column = the thread's index in the
// grid, so the scratch holds align_workers() columns).
template <int BWT, int CM>
__global__ void __launch_bounds__(128, align_blocks(BWT, CM)) align_kernel(ReadsDev rd, ScoreParams sp,
                                                    const uint8_t* __restrict__ genome,
                                                    const uint8_t* __restrict__ mask, int64_t slot0, int64_t nslots,
                                                    PassBuffers pb) {
  __shared__ uint8_t ctab[CM == 1 ? kColourTable : 1];
  if (CM == 1) {
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
    bool masked = false;
    if constexpr (CM == 3) {
      // every cell exact: without masked codes no cell comes near the packed form's floor.  A warp with one
      // masked window runs the general form for all of its windows, not both forms one after the other
      // (3,000 windows of 101 codes, 2 % of the codes masked, -i 3: 198 us, now 109)
      if (s < n) {
        const int64_t slot = slot0 + s;
        const int r = pb.p_read[slot];
        const int64_t win = max(pb.p_diag[slot] - sp.I, -sp.Is);
        masked = window_masked(mask, win, win + rd.lengths[r] + 2 * sp.I);
      }
      masked = __any_sync(0xffffffffu, masked);
    }
    if (s < n) {
      const int64_t slot = pb.round_slots ? (int64_t)pb.round_slots[s] : slot0 + s;
      if constexpr (CM == 2) {
        rows += (unsigned long long)align_one_nuc<BWT, CM == 2>(rd, sp, genome, mask, slot, steal ? tid : s, ns, pb);
      } else if constexpr (CM == 3) {
        if (masked)
          rows += (unsigned long long)align_one<BWT, 0>(rd, sp, genome, mask, slot, steal ? tid : s, ns, pb, ctab);
        else
          rows += (unsigned long long)align_one_nuc<BWT, CM == 2>(rd, sp, genome, mask, slot, steal ? tid : s, ns, pb);
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

}  // namespace sg
