// sw_filter.cuh -- packed 16-bit banded filter over a flat candidate list (sw_filter.cu).
#pragma once

#include "band_core.cuh"
#include "map_kernels.cuh"

namespace sg {

// The banded core of band_core.cuh takes bands of 4, 8 and 16 cells and scores it has bytes for;
// everything else takes filter_core.cuh's.  Both sides at the line, mixed reads at -i 15: 125.6 ms
// with filter_core.cuh, 89.9 ms with band_core.cuh (colour at -i 7: 27.4 and 21.3 ms).
inline int filter_band_registers(int W, const BandConst& c) { return W >= 4 && c.ok ? W / 2 : 0; }

struct FilterJob {
  int64_t n;                    // candidates
  const int32_t* fr;            // read of each candidate
  const int32_t* fd;            // diagonal of each candidate (window start = diag - Is)
  uint8_t* flag;                // out: 1 = passes
  const uint8_t* codes;         // packed reads
  int64_t cstride;
  const int16_t* lengths;
  const uint8_t* genome;
  int W, Is;
  int fm, fx, fo, fe, fthr;
  unsigned long long* counters;  // [2] += cell updates W*2*(L+W-1), [5] += candidates, [6] += L*(2*Is+1)
  const uint8_t* gexp;          // byte-expanded genome (code c -> c * 0x11), code 0
  const uint8_t* rexp;          // read streams (bytes 0xC4 + c * 0x11), rstride bytes per read
  int64_t rstride;
  int min_len;                  // shortest read of the batch (reads shorter than W take another path)
  // may be null; else the candidate count is read from here when the kernel starts (the hit
  // gather's cursor), and n is only an upper bound for the grid
  const unsigned long long* n_dev;
  // may be null; else a zeroed work cursor: the grid is the resident set, and every block takes
  // the next tile of 256 * kFilterTile candidates from it, in list order, until none is left
  unsigned long long* cursor;
  // band registers of the core of band_core.cuh (0: not used), its constants and read streams
  int band_H;
  BandConst band;
  const uint32_t* bs;
  int64_t bwords;  // of a row of bs
  int rows;  // with a cursor: rows of 256 candidates in a block's tile (0 = 8); without: 8, fewer for short lists
};

constexpr int64_t kGexpPad = 4096;   // bytes of padding around a byte-expanded sequence
inline int64_t rexp_stride(int max_len) { return ((int64_t)max_len + 16 + 8 + 15) & ~15LL; }
void launch_expand_genome(const uint8_t* codes, int64_t n_codes, uint8_t* gexp, cudaStream_t st);
void launch_expand_reads(const ReadsDev& rd, uint8_t* rexp, int64_t rstride, cudaStream_t st);

bool filter_dpx_ok(const ScoreParams& sp, int max_len);
void launch_filter_flat_job(const FilterJob& job, const ScoreParams& sp, bool dpx, cudaStream_t st);
// What a selection does with its total on the device (all null: nothing): above cap (the lists' size)
// *status gets bit 2, above limit bit 1; *take becomes the total, or 0 with a status; without one *sum grows
// by it; *most keeps the largest.
struct SelectGate {
  unsigned long long *status, *take, *sum, *most;
  int64_t cap, limit;
};
constexpr int kSelectTile = 4096;  // flag bytes per tile
inline int64_t select_tiles(int64_t ncap) { return (ncap + kSelectTile - 1) / kSelectTile; }
// The flagged of the first n_dev (null: all ncap) candidates, in order, in two launches.  tile: select_tiles(ncap)
// + 1 words, the last of which gets their number; ticket: a zeroed word; flag 16-byte aligned.  The
// second writes those below pcap (the lists' capacity), with p_ub (may be null) their score bounds too.
void launch_select_count(int64_t ncap, const unsigned long long* n_dev, const uint8_t* flag, int64_t* tile,
                         unsigned long long* ticket, const SelectGate& g0, const SelectGate& g1, cudaStream_t st);
void launch_select_write(int64_t ncap, const unsigned long long* n_dev, const uint8_t* flag, const int64_t* tile,
                         const int32_t* fr, const int32_t* fd, int32_t* p_read, int32_t* p_diag, int64_t pcap,
                         const int16_t* ub, int16_t* p_ub, cudaStream_t st);
// Both in one launch of one block, for candidate lists of a capacity up to kSelectSmall (a call of few
// reads: the spare 61,440 places and at most 3,300 expected candidates, so one tile of about 5 us where
// the two launches take 10; a full list would take 30).
constexpr int64_t kSelectSmall = 1 << 16;
void launch_select_small(int64_t ncap, const unsigned long long* n_dev, const uint8_t* flag, const SelectGate& g0,
                         const SelectGate& g1, const int32_t* fr, const int32_t* fd, int32_t* p_read, int32_t* p_diag,
                         int64_t pcap, const int16_t* ub, int16_t* p_ub, cudaStream_t st);
}  // namespace sg
