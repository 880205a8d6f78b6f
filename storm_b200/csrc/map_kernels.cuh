// map_kernels.cuh -- per-pass mapping kernels (one reference sequence x one strand).
#pragma once

#include "common.cuh"

namespace sg {

// Scoring, as the kernels need it.
struct ScoreParams {
  int colour;
  int I;              // -i
  int Is;             // min(-i, 15): SIMD band half-width (main.c:302-313)
  int W;              // filter cells per hit: 2, 4, 8, 16 (run.c:64-101)
  int fm, fx, fo, fe; // filter scores: low bytes of |match|, |mismatch|, |open|, |extend|
  int fthr;           // filter threshold, min(z, 254) (alignment_simd.c:2525-2527)
  int pair[2][4];     // SCALE_SCORE(match|mismatch, level) (alignment.h:30, alignment.c:275-278)
  int gap_open, gap_ext;
  int min_score;      // -t
  // the packed nucleotide alignment (align_one_nuc): used when `packed`; its constants come
  // through the kernel parameters so that the multiply-adds stay multiply-adds
  // (1: in every window; 2, the unit entry points: in windows without masked codes; small: its scores
  // allow it)
  int packed, small;
  uint32_t one;       // 1
  uint32_t open1;     // (gap_open << 13) + 1
  uint32_t open1_tc;  // open1 + (1 << 11) - (1 << 12): a corner-labelled cell as a top gap source
  uint32_t kt, kl;    // 4 (ext - open) - 2^22, 8 (ext - open) - 2^22 (modulo 2^32)
  uint32_t pw[32];    // 2^k
};

// filter width W for the SIMD half-width Is (run.c:64-101), and the scoring of a parameter set
int filter_width(int is);
ScoreParams make_score_params(const stormgpu_params& p);

struct ReadsDev {
  int64_t n;
  const uint8_t* codes;
  int64_t cstride;
  const uint8_t* levels;   // may be null
  int64_t lstride;
  const int16_t* lengths;
  // may be null; else the fused gather visits read order[k] k-th (reads grouped by length, so
  // that the candidate list, and with it the filter's and the alignment's blocks, is too)
  const int32_t* order;
};

struct IndexView {
  const int32_t* first[kMaxSeeds];
  const int32_t* map[kMaxSeeds];
};

struct PassBuffers {
  // filter -> flat list of passing candidates
  int32_t* pstart;      // per read with candidates: first slot
  int32_t* pcount;      // and their number
  // reads with candidates left: the list of this replay (count at active_count[0]) and of the next
  // (active_count[1])
  int32_t* active;
  int32_t* active_next;
  int32_t* active_count;
  int32_t* p_read;      // per slot, reads contiguous
  int32_t* p_diag;      // per slot, ascending within a read
  // align outputs per slot
  int32_t* a_score;
  int32_t* a_bound;
  int16_t* a_pos;       // 4 per slot: best_i, best_j, best_i0, best_j0
  int32_t* a_tblen;
  uint8_t* a_tb;        // tbs bytes per slot (end-to-start order)
  int64_t tbs;
  uint32_t* a_scratch;  // direction bits, see align kernel
  // may be null; else a zeroed work cursor, and the align launch is a persistent grid of
  // align_workers() threads (scratch columns) taking slots from it
  unsigned long long* cursor;
  const int64_t* npass_dev;  // may be null; else the slot count is read from here
  int wave;                  // with a cursor: up to so many slots are left to align_wave_kernel
  int steal;                 // with a cursor: slots a warp takes at a time, a multiple of 32 (0 = 32)
  // Rounds (all null for one round over every slot).  The candidates of a read are aligned in rounds:
  // each takes its next candidates that may still exceed the read's running threshold (see
  // replay_kernel), listed in round_slots, round_count[0] of them (round_count[1]: of the next round); thr[read] holds the replay's running
  // threshold after the rounds before, below which a candidate can no longer be accepted, so that its
  // alignment may stop there; round_cur[2 read], [2 read + 1] the ranks the last selection covered.
  const int16_t* ub;           // may be null; per slot, an upper bound of its score
  int32_t* round_slots;
  unsigned long long* round_count;
  int round;                   // the round of this launch
  int32_t* round_cur;
  int32_t* thr;                // per read; written by the replay of each round
  unsigned long long* cells;   // may be null; += band cells the alignment computed
};

constexpr int kMaxAlignRounds = 6;
// candidates of a read in round k: 8, 16, 32, ...; in the last round all that are left
__host__ __device__ __forceinline__ int align_round_take(int k, int rounds) {
  return k >= rounds ? 0 : k == rounds - 1 ? 0x7fffffff : 8 << k;
}

void launch_reverse_reads(const ReadsDev& in, const uint8_t* first_levels, int colour,
                          uint8_t* rcodes, uint8_t* rlevels, cudaStream_t st);
void launch_init_results(int64_t n, stormgpu_hit* hits, uint8_t* mapped, uint8_t* tb, int64_t tbs,
                         cudaStream_t st);
void launch_align(const ReadsDev& r, const ScoreParams& sp, const uint8_t* genome,
                  const uint8_t* mask, int64_t slot0, int64_t nslots, PassBuffers& pb,
                  cudaStream_t st);
// The same by a warp per slot (no scratch, no rounds), for bands of at most 32 cells: every slot when
// there are at most wave_slots() of them (read from pb.npass_dev when given), else none.  maxL: longest
// read.  The warp form takes 80 us for up to 1,000 windows of 101 codes whatever the band (all at once), 105
// for 2,000, 140 for 3,000 and 153 for 4,000 (colours 95, 140, 178, 202); a thread per slot the same time from 64
// to 8,000 windows: in nucleotides 80 us at -i 3, 93 at 7, 127 at 15, 115 at 1 (crossing near 700, 1,300, 2,600
// and 2,500 windows), in colours 165, 292, 525 and 190 (near 2,700, 5,500, above, and 3,500).  The lines were
// laid where these crossed when the thread form's traceback took longer (88, 111, 149, 190; 223, 260, 432, 735
// us); between the crossing and the line the warp form takes up to 1.3 times as long.
constexpr int wave_slots(const ScoreParams& sp) {
  const int bw = 2 * sp.I + 1;
  return bw > 32 ? 0 : !sp.colour && bw >= 7 && bw <= 15 ? 148 * 8 : 4096;
}
void launch_align_wave(const ReadsDev& r, const ScoreParams& sp, const uint8_t* genome, const uint8_t* mask,
                       int64_t slot0, int64_t nslots, PassBuffers& pb, int maxL, cudaStream_t st);
// scratch columns of a launch_align with a cursor (the threads of its persistent grid)
int64_t align_workers(int64_t nslots, const ScoreParams& sp);
// The candidates of a pass that are aligned, as the filter (and the score bound) left them: reads
// contiguous, each read's diagonals in any order.
struct KeptList {
  int64_t n;                 // or with n_dev (may be null) an upper bound for the grid
  const int64_t* n_dev;
  const int32_t* diag;
  const int16_t* ub;         // may be null
  int32_t* long_list;        // reads with more than kShortSlots candidates (as many as reads), their number (zeroed)
  int32_t* long_count;
  int sort_cap;              // most candidates of a read whose diagonals are not ascending already
};
constexpr int kShortSlots = 64;
// pb.p_diag / pb.ub from the list, ascending within each read; pstart / pcount and the first active
// list; with rounds the first round's slots, `take` per read.  The counts are zeroed by the caller.
// pb.p_read is the list's.
constexpr int64_t kSlotsSmall = 2048;  // up to so many by one launch of one block, else by three
void launch_slot_lists(const KeptList& kl, int16_t* ub, PassBuffers& pb, int take, cudaStream_t st);
// Replay of the active reads (at most n): the whole read (no rounds), or the ranks selected last and
// then the selection of up to `take` candidates for the next round.
void launch_replay(int64_t n, const ScoreParams& sp, int ref_id, int sense, PassBuffers& pb, int take,
                   stormgpu_hit* hits, uint8_t* tb, int64_t tbs, uint8_t* mapped, cudaStream_t st);

}  // namespace sg
