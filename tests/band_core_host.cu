// Test infrastructure: runs the banded core of the filter and of the alignment's score bound
// (storm_b200/csrc/band_core.cuh), compiled for the host, on random cases: as the filter against the
// oracle's filter, as the bound against the same recurrence on plain integers (equal where every
// quality level is 3 and no value leaves the exact range) and against the oracle's alignment score
// (never below it).  Prints the number of cases checked and exits non-zero on the first mismatch.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../storm_b200/csrc/band_core.cuh"

extern "C" {
#include "../oracle/storm_oracle.h"
}

static void pack(const std::vector<int>& c, uint8_t* out) {
  for (size_t i = 0; i < c.size(); ++i) out[i >> 2] |= (uint8_t)(c[i] << ((i & 3) * 2));
}

template <int H, bool WTD>
static int core(const uint8_t* gexp, int64_t pos, const std::vector<int>& read, const std::vector<int>& lev,
                const sg::BandConst& c) {  // the default scores through their immediates, as the kernels
  const int L = (int)read.size();
  const int64_t nw = sg::band_stream_words(L, H);
  std::vector<uint32_t> rs(nw), ws(nw);
  auto nib = [&](int i) { return i < 0 || i >= L ? sg::kBandPad : 4u + (uint32_t)read[i]; };
  auto fac = [&](int i) { return (uint32_t)c.wl[i >= 0 && i < L ? lev[i] : 3]; };
  for (int64_t p = 0; p < nw; ++p) {
    rs[p] = sg::band_stream_word(nib((int)p - H - 1), nib((int)p - H), nib((int)p - 1), nib((int)p));
    ws[p] = fac((int)p - H) | fac((int)p) << 16;
  }
  if (sg::band_is_default_filter(c))
    return sg::band_last_row<H, WTD>(gexp, pos, rs.data(), ws.data(), L, sg::BandFilterDefault(c));
  if (sg::band_is_default_bound(c))
    return sg::band_last_row<H, WTD>(gexp, pos, rs.data(), ws.data(), L, sg::BandBoundDefault(c));
  return sg::band_last_row<H, WTD>(gexp, pos, rs.data(), ws.data(), L, c);
}

template <bool WTD>
static int core_h(int H, const uint8_t* g, int64_t pos, const std::vector<int>& r, const std::vector<int>& lev,
                  const sg::BandConst& c) {
  switch (H) {
  case 2: return core<2, WTD>(g, pos, r, lev, c);
  case 4: return core<4, WTD>(g, pos, r, lev, c);
  case 8: return core<8, WTD>(g, pos, r, lev, c);
  default: return core<12, WTD>(g, pos, r, lev, c);
  }
}

// The bound's recurrence on plain integers, row by row over the diagonals pos .. pos + 2W - 1.
static int plain(const std::vector<int>& g, int64_t pos, const std::vector<int>& r, int W, const int (&pair)[2][4],
                 const std::vector<int>& lev, int o, int e) {
  const int L = (int)r.size(), D = 2 * W, G = (int)g.size(), FL = sg::kBoundFloor - sg::kBoundZero;
  const int ee = e < o ? e : o;
  std::vector<int> M(D, 0), I(D, FL), M1(D), I1(D);
  for (int i = 0; i < L; ++i) {
    for (int d = 0; d < D; ++d) {
      const int64_t j = pos + i + d;
      const int code = j >= 0 && j < G ? g[j] : 0;
      int in = FL;
      if (d + 1 < D) in = std::max(in, std::max(I[d + 1] - ee, M[d + 1] - o));  // from the row above
      if (d > 0) in = std::max(in, std::max(I1[d - 1] - ee, M1[d - 1] - o));    // in the row
      I1[d] = in;
      M1[d] = std::max(M[d] + pair[r[i] != code][lev[i]], in);
    }
    M = M1;
    I = I1;
  }
  int best = -100000;
  for (int d = 0; d < D; ++d) best = std::max(best, M[d]);
  return best;
}

int main(int argc, char** argv) {
  const int cases = argc > 1 ? atoi(argv[1]) : 20000;
  std::mt19937_64 rng(54321);
  const int G = 6000, PAD = 4096;
  std::vector<uint8_t> gbuf(PAD + G / 4 + PAD + 64, 0), mbuf(PAD + G / 4 + PAD + 64, 0x55);
  uint8_t* gen = gbuf.data() + PAD;
  uint8_t* msk = mbuf.data() + PAD;
  std::vector<int> g(G);
  for (int i = 0; i < G; ++i) g[i] = rng() & 3;
  pack(g, gen);
  memset(msk, 0, G / 4);
  std::vector<uint8_t> gxbuf(PAD * 4 + G + PAD * 4, 0);
  uint8_t* gexp = gxbuf.data() + PAD * 4;
  for (int i = 0; i < G; ++i) gexp[i] = (uint8_t)(g[i] * 0x11);
  int nfilter = 0, nequal = 0, nbound = 0, passed = 0, kept = 0;
  for (int t = 0; t < cases; ++t) {
    const int Ls[18] = {1, 2, 4, 7, 8, 15, 16, 17, 24, 31, 33, 35, 49, 50, 76, 100, 150, 251};
    const int L = Ls[rng() % 18];
    const int src = (int)(rng() % (G - L - 80));
    std::vector<int> read(L), lev(L), three(L, 3);
    const double rate = (rng() % 5) * 0.1;
    int at = src;
    const int gap = (int)(rng() % (L + 1)), glen = (int)(rng() % 9) - 4;
    for (int i = 0; i < L; ++i) {
      if (i == gap) at += glen;
      read[i] = (rng() % 1000 < rate * 1000) ? (int)(rng() & 3) : g[std::min(std::max(at + i, 0), G - 1)];
      lev[i] = rng() % 8 ? 3 : (int)(rng() % 4);
    }
    const int64_t stride = ((L + 3) / 4 + 7 + 8) & ~7;
    std::vector<uint8_t> rb(stride + 16, 0), lb(stride + 16, 0);
    pack(read, rb.data());
    pack(lev, lb.data());
    const bool def = rng() % 2;
    const int match = def ? 5 : 1 + (int)(rng() % 9), mism = def ? 4 : 1 + (int)(rng() % 8);
    const int go = def ? 9 : 1 + (int)(rng() % 12), ge = def ? 4 : (int)(rng() % 12);
    const int Ws[3] = {4, 8, 16};
    const int W = Ws[rng() % 3];
    const int64_t pos = (rng() % 3 == 0) ? (int64_t)(rng() % (G + 2 * L)) - L : src - (int64_t)(rng() % (2 * W));
    {
      const int thr = (int)(rng() % 4 ? 5 + rng() % 200 : rng() % 260);
      const sg::BandConst c = sg::band_filter_consts(match, mism, go, ge, thr >= 255 ? 254 : thr);
      if (def && !sg::band_is_default_filter(c)) { printf("default scores have other score bytes\n"); return 1; }
      if (c.ok) {
        const int got = core_h<false>(W / 2, gexp, pos, read, three, c) >= sg::kBandInf;
        const int exp = or_sw_filter(W, L, match, mism, go, ge, thr, gen, pos, rb.data());
        if (got != exp) {
          printf("MISMATCH filter case %d: W=%d L=%d %d/%d/%d/%d thr=%d pos=%lld got=%d exp=%d\n", t, W, L, match, mism,
                 go, ge, thr, (long long)pos, got, exp);
          return 1;
        }
        nfilter++;
        passed += exp;
      }
    }
    const int Is[8] = {1, 3, 5, 7, 10, 15, 20, 23};
    const int I = Is[rng() % 8];
    const int H = I <= 3 ? 2 : I <= 7 ? 4 : I <= 15 ? 8 : 12;
    {
      int pair[2][4];
      for (int l = 0; l < 4; ++l) { pair[0][l] = match * (l + 1) / 4; pair[1][l] = -(mism * (l + 1) / 4); }
      const sg::BandConst c = sg::band_bound_consts(pair, -go, -ge);
      if (def && !sg::band_is_default_bound(c)) { printf("default scores have other score bytes (bound)\n"); return 1; }
      const int tm = 100;
      if (!c.ok) continue;
      const int lim = sg::band_bound_limit(match, mism, L);  // bounds below it are exact
      const int64_t win = pos + (rng() % 3 ? 0 : 2);
      const int b3 = core_h<false>(H, gexp, win, read, three, c) - sg::kBoundZero;
      const int e3 = plain(g, win, read, 2 * H, pair, three, go, ge);
      if (b3 < lim ? b3 != e3 : e3 < lim && lim <= sg::kBoundTop) {
        printf("MISMATCH bound case %d: H=%d L=%d %d/%d/%d/%d win=%lld got=%d exp=%d\n", t, H, L, match, mism, go, ge,
               (long long)win, b3, e3);
        return 1;
      }
      nequal++;
      const int bw = core_h<true>(H, gexp, win, read, lev, c) - sg::kBoundZero;
      stormgpu_params p = {};
      p.match = match; p.mismatch = -mism; p.gap_open = -go; p.gap_extend = -ge; p.allowed_indels = I;
      p.min_score = STORMGPU_MIN_SCORE;
      or_align_out o;
      or_align(&p, rb.data(), lb.data(), L, gen, msk, win, &o);
      const int s = o.score;
      if (bw < lim && bw < s) {
        printf("BOUND BELOW SCORE case %d: H=%d I=%d L=%d %d/%d/%d/%d win=%lld bound=%d score=%d\n", t, H, I, L, match, mism,
               go, ge, (long long)win, bw, s);
        return 1;
      }
      nbound++;
      kept += bw > tm;
    }
  }
  printf("checked filter %d (%d pass) bound %d equal, %d against the alignment (%d above -t)\n", nfilter, passed, nequal,
         nbound, kept);
  return 0;
}
