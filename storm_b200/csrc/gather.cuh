// gather.cuh -- fused hit gather (gather.cu).
#pragma once

#include "map_kernels.cuh"

namespace sg {

struct GatherOut {
  int32_t* fr;                   // flat list: read of each candidate
  int32_t* fd;                   // flat list: diagonal of each candidate
  int64_t cap;                   // capacity of fr / fd
  unsigned long long* counters;  // [3] key lookups, [4] index positions, [7] flat cursor, [8] overflow
  // reads with more positions than a warp holds, with their position counts: up to
  // kSmallGatherCap in (small_list, small_h), more in (big_list, big_h); counts [0] big, [2] small
  int32_t* big_list;
  int32_t* big_h;
  int32_t* small_list;
  int32_t* small_h;
  int32_t* big_count;
  unsigned long long* cursor;    // zeroed work cursor of the fused gather (reads taken so far)
  int reads_per_steal;           // reads a warp takes from the cursor at a time (>= 1)
  int warp_cap;                  // index positions a warp holds in shared memory, <= kMaxWarpCap;
                                 // reads with more go to the block kernel
};

constexpr int kMaxWarpCap = 1536;


// The seed family travels with every launch (a kernel parameter), so that mapping calls with
// different seed families can run concurrently on different streams.
void launch_gather_fused(const ReadsDev& rd, const IndexView& ix, int I, const GatherOut& go, const SeedSet& seeds,
                         cudaStream_t st);
// Reads the warp gather handed on, with their position counts (with n_dev, which may be null, the
// number is read from there when the kernel starts and n is only an upper bound), taken from the
// zeroed `cursor` by a persistent grid; reads with too many positions for the launch are appended to
// (above, above_h), counted in above_count.
struct GatherList {
  const int32_t* read;
  const int32_t* h;
  int64_t n;
  const int32_t* n_dev;
  unsigned long long* cursor;
  int32_t* above;
  int32_t* above_h;
  int32_t* above_count;
};

// sorted in shared memory: reads of at most kSmallGatherCap positions (small), else kSortGatherCap
constexpr int kSmallGatherCap = 4096;
constexpr int kSortGatherCap = 65535;
void launch_gather_sort(const ReadsDev& rd, const IndexView& ix, int I, int64_t n_codes, const GatherList& l, bool small,
                        const GatherOut& go, const SeedSet& seeds, cudaStream_t st);
// in global memory: reads of at most `cap` positions, at most `grid` blocks (gather_huge_grid() are
// useful), scratch of cap words each
void launch_gather_huge(const ReadsDev& rd, const IndexView& ix, int I, int64_t n_codes, const GatherList& l,
                        int32_t* scratch, int cap, int64_t grid, const GatherOut& go, const SeedSet& seeds,
                        cudaStream_t st);
int64_t gather_huge_grid();

}  // namespace sg
