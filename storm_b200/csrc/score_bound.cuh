// score_bound.cuh -- upper bound of a passing candidate's alignment score (score_bound.cu).
#pragma once

#include "band_core.cuh"
#include "map_kernels.cuh"

namespace sg {

constexpr int kMaxBoundIndels = 23;  // widest band instantiated: 24 cells per step, 48 diagonals

// Registers of the band that covers the 2I + 1 diagonals of -i I.
inline int bound_registers(int I) { return I <= 3 ? 2 : I <= 7 ? 4 : I <= 15 ? 8 : 12; }

// Read streams of a band of H registers (band_core.cuh): row r of rs, `words` words, and with
// levels the factor stream ws (may be null) from the per-level factors wl.
void launch_band_streams(const ReadsDev& rd, int H, int64_t words, uint32_t* rs, uint32_t* ws, const BandConst& c,
                         cudaStream_t st);

struct BoundJob {
  int64_t n;                 // candidates, or with n_dev (may be null) an upper bound of them
  const int64_t* n_dev;
  const int32_t* read;       // read and diagonal of each candidate
  const int32_t* diag;
  const int16_t* lengths;
  const uint8_t* gexp;       // byte-expanded genome, code 0
  const uint32_t* rs;        // read streams
  const uint32_t* ws;        // factor streams; null: every quality level is 3
  int64_t words;             // of a row of rs / ws
  int H, I, Is;
  int min_score;             // -t
  int match, mismatch;       // scores at quality level 3, positive (band_bound_limit)
  uint8_t* flag;             // out: 1 = may score above -t
  int16_t* ub;               // out: the bound (32767: none)
};
void launch_score_bound(const BoundJob& job, const BandConst& c, cudaStream_t st);

}  // namespace sg
