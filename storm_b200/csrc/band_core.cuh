// band_core.cuh -- one banded affine-gap DP per thread with the score added on the FMA pipe, used
// by the banded filter (sw_filter.cu) and by the score bound of the full alignment
// (score_bound.cu).  Host-and-device, so that the kernels' code is checked on a CPU.
//
// The band has W = 2H cells on every anti-diagonal step, in H registers of two 16-bit cells
// (register j: cells j and j + H).  A pair of steps moves the band one read code (even step) and
// one genome code (odd step); cell k of pair p is at read position p - W + 1 + k.  Per cell
//   D = M[l-2] + score(read code, genome code)                  (one fma.rn.f16x2)
//   J = max(g[l-1], g[l-1] of the neighbour, floor + open)      (gap state + open)
//   M = max(J - open, D)      g = max(J - ext, D)               (one add-max each)
// which is M = max(D, I), I = max over {cell, neighbour} of (I - ext, M - open), not below the
// floor: M >= I, so with ext <= open the gap state after this step is max(I - ext, D - open), kept
// with open added so that neither M nor the gap state needs a subtraction of its own.
//
// Cells are 16-bit integers that are also fp16 numbers: inside one binade the bit pattern of an
// fp16 number counts its value in units of its last place, so fp16 additions (FMA pipe) and DPX
// add-max / max (ALU pipe) work on the same registers exactly.  Two placements of the zero:
//   * filter: zero at pattern 0x7C00 - (threshold + 1).  The cell value threshold + 1 is then 65536,
//     which rounds to infinity, and infinity plus any score is infinity: a cell that passes the
//     threshold marks its diagonal to the end of the read, and no running maximum is kept; the
//     cells are looked at once, after the last row.  Exact for any threshold up to 254.
//   * bound: zero at 1280.0 (unit 1): values -248 .. 767 exact, see score_bound.cu.
// The score: nibbles 4 + c (read) and g (genome) differ by 1..7, 4 where the codes are equal, and
// one prmt turns the differences of four cells into four bytes (match or mismatch byte).  A byte
// serves as the high byte of an fp16 number; its low byte is then the byte of another cell (or 0
// after the shift that moves the other two cells up).  That noise is harmless where factor * number
// rounds to the wanted score whatever the low byte: band_consts looks for two such bytes and a
// factor, and scores that have none (above 7 or so) take the kernels of filter_core.cuh.
// The match byte is negative and the mismatch byte positive (the factor is negative): read nibble 11
// then picks, whatever the genome code, the sign of a mismatch byte, a score of zero.  The read is
// padded with it on both sides: a row of zero scores hands every cell down its diagonal unchanged and
// gaps cannot raise the maximum, so the cells before the read stay zero, those after it keep their
// last row's value, and one loop of whole blocks without masks runs the candidate, reads shorter
// than the band included.  (Masks on the first and last W pairs save 4 % of the cells, 97.5 against
// 102.4 ms before the immediates below, for code five times as long and a case apart for short reads.)
// So a register of two cells costs 3 add-max / max and half a prmt on the ALU pipe, where
// filter_core.cuh's form costs 4.5 (three maxima, a prmt, half a running-maximum fold): 8.5 against
// 6.1 T cell updates/s on the mixed workload's reads, ALU pipe at 81 % of its peak before the
// immediates (the rest: operand reads of three-register instructions).
#pragma once

#include <cmath>
#include <cstdint>
#include <cuda_fp16.h>

#include "filter_core.cuh"

namespace sg {

struct BandConst {
  uint32_t t0, t1;  // prmt table: byte 4 the match byte, bytes 1-3 and 5-7 the mismatch byte
  uint32_t k;       // factor (both halves) at quality level 3
  uint32_t z;       // zero (both halves)
  uint32_t fl;      // floor + open
  uint32_t no, ne;  // -open, -min(ext, open)
  int ok;           // the scores have such bytes
  uint16_t wl[4];   // factor per quality level (bound)
};

constexpr int kBandInf = 0x7C00;
constexpr int kBoundZero = 0x6500;   // 1280.0
constexpr int kBoundFloor = 0x6408;  // value -248; -255 is the binade's lowest
constexpr int kBoundTop = 767;       // largest exact value

SG_HD uint32_t band_fma(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__)
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
#else
  uint32_t out = 0;
  for (int h = 0; h < 2; ++h) {
    double v[3];
    const uint32_t in[3] = {a, b, c};
    for (int i = 0; i < 3; ++i) {
      __half_raw r;
      r.x = (unsigned short)(in[i] >> (16 * h));
      v[i] = (double)__half2float(__half(r));
    }
    const __half_raw q = __half_raw(__double2half(v[0] * v[1] + v[2]));  // exact in double, one rounding
    out |= (uint32_t)q.x << (16 * h);
  }
  return out;
#endif
}

SG_HD void ldg128(const uint32_t* p, uint32_t (&v)[4]) {
#if defined(__CUDA_ARCH__)
  const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
#else
  for (int i = 0; i < 4; ++i) v[i] = p[i];
#endif
}

__host__ __device__ constexpr int band_block(int H) { return H == 2 ? 4 : H; }  // pairs of a main block: a multiple of 4 and of H

// Read stream of a band of H registers: word p (the codes entering at pair p) holds the nibbles of
// positions p - H - 1, p - H, p - 1 and p: 4 + code inside the read, 11 outside it.
constexpr uint32_t kBandPad = 11;
__host__ __device__ inline int64_t band_stream_words(int max_len, int H) {
  const int bp = band_block(H);
  return ((int64_t)max_len + 2 * H - 1 + bp - 1) / bp * bp;
}
SG_HD uint32_t band_stream_word(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return a | (b << 4) | (c << 8) | (d << 12);
}

template <int H>
struct Band {
  static constexpr int W = 2 * H;
  static constexpr int BP = band_block(H);
  static constexpr int NH = (H + 3) / 4;  // genome words an entry reaches back
  static_assert(H % 2 == 0 && BP % 4 == 0 && BP % H == 0, "register count");
  uint32_t M1[H], M2[H], G[H];
  uint32_t ra[H], gb[H];  // entries of four codes: read entry i in slot i mod H, genome entry x in slot x mod H
  uint32_t wt[H];         // factors of cells (j, j + H), weighted form only
};

// One step; Q = pair mod H.
template <int H, bool ODD, int Q, bool WTD, class C>
SG_HD void band_step(Band<H>& b, const C& c) {
  uint32_t sc[H], J[H];
#pragma unroll
  for (int q = 0; q < H / 2; ++q) {
    const uint32_t sel = b.ra[(Q + 1 + 2 * q) % H] - b.gb[((ODD ? Q : Q - 1) - 2 * q + 2 * H) % H];
    const uint32_t x = prmt(c.t0, c.t1, sel);
    sc[2 * q + 1] = x;
    sc[2 * q] = x << 8;
  }
#pragma unroll
  for (int j = 0; j < H; ++j) {
    uint32_t nb;
    if (ODD) nb = j > 0 ? b.G[j - 1] : prmt(c.fl, b.G[H - 1], 0x5410);
    else     nb = j < H - 1 ? b.G[j + 1] : prmt(b.G[0], c.fl, 0x5432);
    J[j] = __vimax3_s16x2(b.G[j], nb, c.fl);
  }
#pragma unroll
  for (int j = 0; j < H; ++j) {
    const uint32_t w = WTD ? b.wt[(Q + 1 + j) % H] : c.k;
    const uint32_t D = band_fma(sc[j], w, b.M2[j]);
    b.G[j] = __viaddmax_s16x2(J[j], c.ne, D);
    b.M2[j] = b.M1[j];
    b.M1[j] = __viaddmax_s16x2(J[j], c.no, D);
  }
}

template <int H, int Q, bool WTD, class C>
SG_HD void band_pair(Band<H>& b, const C& c, uint32_t rs, uint32_t ws, uint32_t gg) {
  b.ra[(Q + H - 1) % H] = rs;
  if (WTD) b.wt[Q % H] = ws;
  band_step<H, false, Q % H, WTD>(b, c);
  b.gb[Q % H] = gg;
  band_step<H, true, Q % H, WTD>(b, c);
}

// Genome words from code x0 on: byte-expanded codes (c * 0x11) regrouped so that byte x holds the
// nibbles of codes x and x - 1.
struct BandGenome {
  const uint32_t* w;
  uint32_t raw, prev, sel;
  SG_HD void init(const uint8_t* gexp, int64_t x0) {
    w = reinterpret_cast<const uint32_t*>(gexp) + (x0 >> 2);
    sel = funnel_sel((uint32_t)(x0 & 3));
    raw = ldg32(w);
    ++w;
    prev = 0;
  }
  SG_HD uint32_t next() {
    const uint32_t n = ldg32(w);
    ++w;
    const uint32_t g = prmt(raw, n, sel);
    raw = n;
    const uint32_t sh = prmt(prev, g, 0x6543);
    prev = g;
    return (g & 0x0F0F0F0Fu) | (sh & 0xF0F0F0F0u);
  }
};

// entry of code X: bytes X and X - H of the words (word 0 holds codes 0..3)
template <int H, int X, int NW>
SG_HD uint32_t band_entry(const uint32_t (&t)[NW]) {
  constexpr int Y = X - H;
  static_assert(Y >= 0 && X / 4 < NW, "entry outside the words");
  return prmt(t[X / 4], t[Y / 4], (uint32_t)(X % 4) | ((uint32_t)(4 + Y % 4) << 4));
}

// Pairs K .. NP - 1 of a block; t holds the block's genome words after NH words of history; rs / ws
// the entering read and factor words.
template <int H, int K, int NP, bool WTD, int NW, int NR, int NS, class C>
SG_HD void band_run(Band<H>& b, const C& c, const uint32_t (&t)[NW], const uint32_t (&rs)[NR],
                    const uint32_t (&ws)[NS]) {
  if constexpr (K < NP) {
    band_pair<H, K, WTD>(b, c, rs[K], WTD ? ws[WTD ? K : 0] : 0u, band_entry<H, 4 * Band<H>::NH + K, NW>(t));
    band_run<H, K + 1, NP, WTD, NW, NR, NS>(b, c, t, rs, ws);
  }
}

template <int H, int X, int NW>
SG_HD void band_fill(Band<H>& b, const uint32_t (&t)[NW]) {  // genome entries X .. W - 1 (code 0: the window's first)
  if constexpr (X < 2 * H) {
    b.gb[X % H] = band_entry<H, X, NW>(t);
    band_fill<H, X + 1, NW>(b, t);
  }
}

// n stream words from p on (16-byte aligned)
template <int N, int M>
SG_HD void band_load(const uint32_t* p, uint32_t (&v)[M]) {
#pragma unroll
  for (int m = 0; m < N / 4; ++m) {
    uint32_t q[4];
    ldg128(p + 4 * m, q);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[4 * m + i] = q[i];
  }
}

// One candidate: the largest cell of the last read row, as a pattern (see the two placements).
// gexp: byte-expanded genome (code c -> c * 0x11) at code 0, 4-byte aligned, readable from pos to
// pos + L + 3W + 8; rs: the read's stream, 16-byte aligned, band_stream_words(L, H) words; ws: its
// factor stream (weighted form): word p the factors of positions p - H and p.
template <int H, bool WTD, class C>
SG_HD int band_last_row(const uint8_t* __restrict__ gexp, int64_t pos, const uint32_t* __restrict__ rs,
                        const uint32_t* __restrict__ ws, int L, const C& c) {
  constexpr int W = 2 * H, NH = Band<H>::NH, BP = Band<H>::BP, NB = BP / 4, NP4 = W / 4;
  Band<H> b;
#pragma unroll
  for (int j = 0; j < H; ++j) {
    b.M1[j] = c.z; b.M2[j] = c.z; b.G[j] = c.z;
    b.ra[j] = kBandPad * 0x1111u;
    b.gb[j] = 0;
    b.wt[j] = c.k;
  }
  BandGenome gs;
  gs.init(gexp, pos);
  uint32_t hist[NH];
  {  // codes pos .. pos + W - 1
    uint32_t t[NP4];
#pragma unroll
    for (int m = 0; m < NP4; ++m) t[m] = gs.next();
    band_fill<H, H + 1, NP4>(b, t);
#pragma unroll
    for (int m = 0; m < NH; ++m) hist[m] = t[NP4 - NH + m];
  }
  const int n = L + W - 1;  // after that many pairs every cell is on the last row or below it
#pragma unroll 1
  for (int p = 0; p < n; p += BP) {
    uint32_t t[NH + NB], r[BP], w[WTD ? BP : 4];
#pragma unroll
    for (int m = 0; m < NH; ++m) t[m] = hist[m];
#pragma unroll
    for (int m = 0; m < NB; ++m) t[NH + m] = gs.next();
    band_load<BP>(rs + p, r);
    if (WTD) band_load<WTD ? BP : 4>(ws + p, w);
    band_run<H, 0, BP, WTD, NH + NB, BP, (WTD ? BP : 4)>(b, c, t, r, w);
#pragma unroll
    for (int m = 0; m < NH; ++m) hist[m] = t[NB + m];
  }
  uint32_t mx = 0x80008000u;
#pragma unroll
  for (int j = 0; j < H; ++j) mx = __vimax3_s16x2(mx, b.M1[j], b.M2[j]);
  const int hi = (int)(int16_t)(mx >> 16), lo = (int)(int16_t)(mx & 0xFFFFu);
  return hi > lo ? hi : lo;
}

// ------------------------------------------------------------------------------ constants (host)

inline double band_half(unsigned pattern) {
  __half_raw r;
  r.x = (unsigned short)pattern;
  return (double)__half2float(__half(r));
}
inline unsigned band_half_bits(double v) { return __half_raw(__double2half(v)).x; }

// The two bytes and the (negative) factor for scores +match / -mismatch counted in units of `unit`:
// whatever the low byte (0 or one of the two bytes), factor * number is within 0.45 units of the
// score, and within 0.1 units of zero when the high byte is 0.  The choice with the largest margin.
inline bool band_score_bytes(int match, int mismatch, double unit, unsigned* hm, unsigned* hx, unsigned* k) {
  if (match < 1 || mismatch < 1 || match > 15 || mismatch > 15) return false;
  double best = 0.05;
  bool found = false;
  for (unsigned m = 0x04; m < 0x30; ++m)
    for (unsigned x = 0x04; x < 0x30; ++x) {
      const unsigned low[3] = {0, m | 0x80, x};
      double mlo = 1e30, mhi = 0, xlo = 1e30, xhi = 0;
      for (unsigned n : low) {
        const double vm = band_half(m << 8 | n), vx = band_half(x << 8 | n);
        mlo = std::fmin(mlo, vm); mhi = std::fmax(mhi, vm);
        xlo = std::fmin(xlo, vx); xhi = std::fmax(xhi, vx);
      }
      // factors with every product within half a unit
      const double flo = std::fmax((match - 0.5) * unit / mlo, (mismatch - 0.5) * unit / xlo);
      const double fhi = std::fmin((match + 0.5) * unit / mhi, (mismatch + 0.5) * unit / xhi);
      if (!(flo < fhi) || flo > 60000.0) continue;
      const unsigned kb = band_half_bits(0.5 * (flo + fhi));
      const double f = band_half(kb);
      if (!(f < 65000.0) || f < 1.0 / 4096 || f * band_half(m | 0x80) > 0.1 * unit) continue;
      const double margin = std::fmin(std::fmin(f * mlo / unit - (match - 0.5), match + 0.5 - f * mhi / unit),
                                      std::fmin(f * xlo / unit - (mismatch - 0.5), mismatch + 0.5 - f * xhi / unit));
      if (margin > best) {
        best = margin;
        *hm = m | 0x80; *hx = x; *k = kb | 0x8000u;
        found = true;
      }
    }
  return found;
}

inline void band_table(unsigned hm, unsigned hx, BandConst* c) {
  c->t0 = hx << 8 | hx << 16 | hx << 24;
  c->t1 = hm | hx << 8 | hx << 16 | hx << 24;
}

// The filter's constants: scores as absolute values (low bytes), threshold at most 254.
inline BandConst band_filter_consts(int fm, int fx, int fo, int fe, int fthr) {
  BandConst c = {};
  unsigned hm = 0, hx = 0, k = 0;
  c.ok = fthr >= 0 && fthr <= 254 && band_score_bytes(fm, fx, 32.0, &hm, &hx, &k) ? 1 : 0;
  if (!c.ok) return c;
  band_table(hm, hx, &c);
  c.k = k * 0x10001u;
  const uint32_t z = (uint32_t)(kBandInf - (fthr + 1));
  c.z = z * 0x10001u;
  c.fl = (z + (uint32_t)fo) * 0x10001u;
  c.no = (uint32_t)(uint16_t)(-fo) * 0x10001u;
  c.ne = (uint32_t)(uint16_t)(-(fe < fo ? fe : fo)) * 0x10001u;
  return c;
}

// The constants of the default scores (5, -4, -9, -4; alignment.h:24-28) as immediates: a cell's four
// instructions then read two or three registers each instead of up to three and a constant, and
// the register file, not only the ALU pipe, limits them (4,000 mixed reads at -i 15: filter 99.6 ms
// with run-time constants, 88.2-91.8 ms with these).  Other scores run the same kernels on a
// BandConst; band_is_default compares, so that these follow band_consts' choice.
struct BandFilterDefault {
  static constexpr uint32_t t0 = 0x18181800u, t1 = 0x18181899u, k = 0xfb84fb84u, no = 0xfff7fff7u, ne = 0xfffcfffcu;
  uint32_t z, fl;  // by the threshold
  SG_HD BandFilterDefault(const BandConst& c) : z(c.z), fl(c.fl) {}
};
struct BandBoundDefault {
  static constexpr uint32_t t0 = 0x10101000u, t1 = 0x10101091u, k = 0xef8bef8bu, no = 0xfff7fff7u, ne = 0xfffcfffcu;
  static constexpr uint32_t z = 0x65006500u, fl = 0x64116411u;
  SG_HD BandBoundDefault(const BandConst&) {}
};
inline bool band_is_default_filter(const BandConst& c) {
  using D = BandFilterDefault;
  return c.ok && c.t0 == D::t0 && c.t1 == D::t1 && c.k == D::k && c.no == D::no && c.ne == D::ne;
}
inline bool band_is_default_bound(const BandConst& c) {
  using D = BandBoundDefault;
  return c.ok && c.t0 == D::t0 && c.t1 == D::t1 && c.k == D::k && c.no == D::no && c.ne == D::ne && c.z == D::z &&
         c.fl == D::fl;
}

// The bound's constants: pair scores per quality level (pair[0] match, pair[1] mismatch), gap scores
// (negative).  A level below 3 gets a factor whose products round to at least that level's scores.
inline BandConst band_bound_consts(const int (&pair)[2][4], int gap_open, int gap_ext) {
  BandConst c = {};
  unsigned hm = 0, hx = 0, k = 0;
  const int a = pair[0][3], b = -pair[1][3], o = -gap_open, e = -gap_ext;
  c.ok = o >= 1 && o <= 255 && e >= 0 && e <= 255 && band_score_bytes(a, b, 1.0, &hm, &hx, &k) ? 1 : 0;
  if (!c.ok) return c;
  band_table(hm, hx, &c);
  c.k = k * 0x10001u;
  c.z = (uint32_t)kBoundZero * 0x10001u;
  c.fl = (uint32_t)(kBoundFloor + o) * 0x10001u;
  c.no = (uint32_t)(uint16_t)(-o) * 0x10001u;
  c.ne = (uint32_t)(uint16_t)(-(e < o ? e : o)) * 0x10001u;
  c.wl[3] = (uint16_t)k;
  const unsigned low[3] = {0, hm, hx};
  for (int l = 0; l < 3; ++l) {
    int best = 1 << 20;
    for (int s = 1; s <= 512; ++s) {
      const unsigned fb = band_half_bits(band_half(k) * s / 512.0);
      const double f = band_half(fb);
      int over = 0;
      for (unsigned n : low) {
        const double m = f * band_half(hm << 8 | n), x = f * band_half(hx << 8 | n);
        // the sum with a whole number rounds to nearest; keep 0.02 away from ties
        const int rm = (int)std::floor(m - 0.02 + 0.5), rx = (int)std::floor(x - 0.02 + 0.5);
        if (rm < pair[0][l] || rx < pair[1][l]) { over = 1 << 20; break; }
        over += rm - pair[0][l] + rx - pair[1][l];
      }
      if (over < best) { best = over; c.wl[l] = (uint16_t)fb; }
    }
    if (best >= 1 << 20) c.ok = 0;
  }
  return c;
}

// A bound below this is exact (and so never below the score) for a read of L codes.  A cell above
// kBoundTop is in a binade of unit 2 (each step may round down by 1) or infinite; it loses at most
// mismatch + 1 on each row of its diagonal until it is back below, so a path that was ever there
// ends at this value or above.
SG_HD int band_bound_limit(int match, int mismatch, int L) {
  const int r0 = kBoundTop / match;  // rows in which no path exceeds kBoundTop
  return L <= r0 ? kBoundTop + 1 : kBoundTop - (mismatch + 1) * (L - r0);
}

}  // namespace sg
