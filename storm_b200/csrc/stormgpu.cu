// stormgpu.cu -- the C ABI of include/stormgpu.h: context, reference upload, index build,
// and the mapping pipeline (per reference sequence, per strand: hit gather -> filter ->
// full alignment -> top-4 replay), plus the unit-level entry points used by the tests.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "index_build.cuh"
#include "map_kernels.cuh"
#include "scan.cuh"
#include "sw_filter.cuh"
#include "score_bound.cuh"
#include "gather.cuh"
#include "radix.cuh"
#include "context.cuh"

static thread_local char g_err[1024];
thread_local sg::WorkBudget* sg::g_work_budget = nullptr;

void sg_set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

extern "C" const char* stormgpu_version(void) { return "storm-b200 0.1 (sm_100a)"; }
extern "C" const char* stormgpu_last_error(void) { return g_err; }

extern "C" int stormgpu_device_available(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) { cudaGetLastError(); return 0; }
  return n > 0 ? 1 : 0;
}

namespace {

using namespace sg;

// seed.c:25-135: ';'-separated patterns of '#'/'1' (care) and '-'/'0' (don't care), each with
// an optional ":p1 p2,p3" list of read positions.
int parse_seeds(const char* list, SeedSet* out) {
  memset(out, 0, sizeof(*out));
  if (!list) return STORMGPU_EINVAL;
  std::string s(list);
  size_t p = 0;
  while (p <= s.size()) {
    size_t e = s.find(';', p);
    if (e == std::string::npos) e = s.size();
    std::string tok = s.substr(p, e - p);
    p = e + 1;
    if (tok.empty()) { if (e == s.size()) break; continue; }
    if (out->n >= kMaxSeeds) return STORMGPU_EINVAL;
    SeedDev& sd = out->s[out->n];
    size_t colon = tok.find(':');
    std::string pat = tok.substr(0, colon);
    if (pat.empty() || (int)pat.size() > kMaxSpan) return STORMGPU_EINVAL;
    sd.span = (int)pat.size();
    for (int i = 0; i < sd.span; ++i) {
      char c = pat[i];
      if (c == '#' || c == '1') sd.care[sd.n_care++] = (int8_t)i;
      else if (c != '-' && c != '0') return STORMGPU_EINVAL;
    }
    sd.weight = sd.n_care;
    if (sd.weight == 0 || sd.weight > 15) return STORMGPU_EINVAL;
    if (colon != std::string::npos && tok.size() - colon > 1) {
      std::string rest = tok.substr(colon + 1);
      int v;
      if (sscanf(rest.c_str(), "%d", &v) == 1) {
        char* save = nullptr;
        std::vector<char> buf(rest.begin(), rest.end());
        buf.push_back(0);
        for (char* t = strtok_r(buf.data(), ", ", &save); t; t = strtok_r(nullptr, ", ", &save)) {
          if (sscanf(t, "%d", &v) != 1 || sd.n_positions >= kMaxPositions) break;
          sd.positions[sd.n_positions++] = (int16_t)v;
        }
      }
    }
    out->n++;
    if (e == s.size()) break;
  }
  return out->n > 0 ? 0 : STORMGPU_EINVAL;
}

}  // namespace

namespace sg {

int filter_width(int is) { return is <= 1 ? 2 : is <= 3 ? 4 : is <= 7 ? 8 : 16; }

ScoreParams make_score_params(const stormgpu_params& p) {
  ScoreParams sp;
  memset(&sp, 0, sizeof(sp));
  sp.colour = p.colour;
  sp.I = p.allowed_indels;
  sp.Is = p.allowed_indels < 15 ? p.allowed_indels : 15;
  sp.W = filter_width(sp.Is);
  sp.fm = std::abs(p.match) & 0xff;
  sp.fx = std::abs(p.mismatch) & 0xff;
  sp.fo = std::abs(p.gap_open) & 0xff;
  sp.fe = std::abs(p.gap_extend) & 0xff;
  unsigned z = (unsigned)p.min_score_filter;
  sp.fthr = z >= 255u ? 254 : (int)z;
  for (int l = 0; l < 4; ++l) {
    sp.pair[0][l] = (int)(((p.match) * (l + 1) + 0.) / 4);     // SCALE_SCORE, alignment.h:30
    sp.pair[1][l] = (int)(((p.mismatch) * (l + 1) + 0.) / 4);
  }
  sp.gap_open = p.gap_open;
  sp.gap_ext = p.gap_extend;
  sp.min_score = p.min_score;
  // packed cells (align_one_nuc): scores and penalties below 256 in magnitude, at most 200
  // indels, a read's largest gain below 48000 (a floored cell stays under MIN_SCORE) and -t
  // minus that gain above the floor's score -2^16
  int maxpair = 0;
  for (int l = 0; l < 4; ++l) maxpair = std::max({maxpair, std::abs(sp.pair[0][l]), std::abs(sp.pair[1][l])});
  sp.small = !p.colour && p.allowed_indels >= 0 && p.allowed_indels <= 200 && maxpair <= 255 &&
             std::abs(p.gap_open) <= 255 && std::abs(p.gap_extend) <= 255 &&
             (int64_t)STORMGPU_MAX_READ_LEN * maxpair < 48000;
  sp.packed = sp.small && (int64_t)p.min_score - (int64_t)STORMGPU_MAX_READ_LEN * maxpair > -60000;
  sp.one = 1u;
  sp.open1 = (uint32_t)p.gap_open * 8192u + 1u;
  sp.open1_tc = sp.open1 + (1u << 11) - (1u << 12);
  const uint32_t dx = (uint32_t)(p.gap_extend - p.gap_open);
  sp.kt = 4u * dx - (1u << 22);
  sp.kl = 8u * dx - (1u << 22);
  for (int k = 0; k < 32; ++k) sp.pw[k] = 1u << k;
  return sp;
}

}  // namespace sg



extern "C" int stormgpu_open(const stormgpu_params* params, const char* seeds, stormgpu_ctx** out) {
  if (!params || !out) { sg_set_error("null argument"); return STORMGPU_EINVAL; }
  *out = nullptr;
  SeedSet ss;
  if (parse_seeds(seeds, &ss) != 0) { sg_set_error("invalid seed list \"%s\"", seeds ? seeds : "(null)"); return STORMGPU_EINVAL; }
  if (params->allowed_indels < 0 || params->allowed_indels > STORMGPU_MAX_INDELS) { sg_set_error("allowed_indels out of range"); return STORMGPU_EINVAL; }
  if (params->min_score < STORMGPU_MIN_SCORE) { sg_set_error("min_score below MIN_SCORE is not supported"); return STORMGPU_EINVAL; }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    sg_set_error("no CUDA device available: the mapping path runs on the GPU only");
    return STORMGPU_ECUDA;
  }
  if (params->device < 0 || params->device >= ndev) { sg_set_error("bad device ordinal"); return STORMGPU_EINVAL; }
  SG_CUDA(cudaSetDevice(params->device));
  {
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, params->device) == cudaSuccess) {
      uint64_t keep = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    cudaGetLastError();
  }
  stormgpu_ctx* c = new stormgpu_ctx();
  c->p = *params;
  c->seeds = ss;
  memset(&c->stats, 0, sizeof(c->stats));
  if (cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) != cudaSuccess) {
    delete c;
    sg_set_error("cudaStreamCreate failed");
    return STORMGPU_ECUDA;
  }
  for (auto& e : c->ev) cudaEventCreate(&e);
  for (auto& e : c->rev) cudaEventCreate(&e);
  if (const char* g = getenv("STORMGPU_GRAPHS")) c->graphs = atoi(g) != 0;
  *out = c;
  return 0;
}

extern "C" int stormgpu_set_graphs(stormgpu_ctx* c, int enable) {
  if (!c) { sg_set_error("null argument"); return STORMGPU_EINVAL; }
  c->graphs = enable != 0;
  return 0;
}

// Every buffer that a mapping call grows for itself (what its working memory limit counts).
static void release_work(stormgpu_ctx* c) {
  c->rcodes.release(); c->rlevels.release();
  c->pstart.release(); c->pcount.release(); c->p_read.release(); c->p_diag.release();
  c->big_list.release(); c->big_h.release(); c->small_list.release(); c->small_h.release();
  c->huge_list.release(); c->huge_h.release();
  c->a_score.release(); c->a_bound.release(); c->a_tblen.release(); c->big_tmp.release();
  c->a_pos.release(); c->a_tb.release(); c->scratch.release(); c->counters.release();
  c->foff.release(); c->fr.release(); c->fd.release(); c->flag.release();
  c->rexp.release();
  c->q_read.release(); c->q_diag.release(); c->q_ub.release(); c->k_ub.release(); c->p_ub.release();
  c->k_diag.release(); c->long_list.release(); c->bstream.release(); c->wstream.release();
  c->ord.release(); c->ord_tmp.release();
  c->thr.release(); c->active.release(); c->round_cur.release(); c->round_slots.release();
  c->work.used = 0;
}

extern "C" void stormgpu_close(stormgpu_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->p.device);
  cudaStreamSynchronize(c->st);
  if (c->owns_refs)
    for (auto& r : c->refs) {
      cudaFree(r.d_codes_alloc);
      cudaFree(r.d_mask_alloc);
      cudaFree(r.d_gexp_alloc);
      for (auto& ix : r.idx) { cudaFree(ix.first); cudaFree(ix.map); }
    }
  release_work(c);
  c->fcodes.release(); c->flevels.release(); c->first_levels.release(); c->lengths.release();
  c->hits.release(); c->tb.release(); c->mapped.release();
  c->gm_k0.release(); c->gm_v0.release(); c->gm_k1.release(); c->gm_v1.release(); c->gm_tmp.release();
  c->gm_base.release();
  for (auto& e : c->gev) cudaEventDestroy(e);
  for (auto& e : c->ev) cudaEventDestroy(e);
  for (auto& e : c->rev) cudaEventDestroy(e);
  cudaStreamDestroy(c->st);
  delete c;
}

extern "C" int stormgpu_add_reference(stormgpu_ctx* c, const uint8_t* codes, const uint8_t* mask,
                                      int64_t n_codes, const int32_t* rs, const int32_t* re,
                                      int32_t n_regions) {
  if (!c || !codes || n_codes < 0 || (n_regions > 0 && (!rs || !re))) { sg_set_error("bad reference arguments"); return STORMGPU_EINVAL; }
  if (n_codes >= INT32_MAX) { sg_set_error("reference sequence longer than 2^31 codes"); return STORMGPU_EINVAL; }
  SG_CUDA(cudaSetDevice(c->p.device));
  RefSeq r;
  r.n = n_codes;
  const int64_t nb = (n_codes + 3) / 4;
  const int64_t tot = nb + 2 * kPadBytes + 16;
  SG_CUDA(cudaMalloc(&r.d_codes_alloc, tot));
  SG_CUDA(cudaMalloc(&r.d_mask_alloc, tot));
  r.d_codes = r.d_codes_alloc + kPadBytes;
  r.d_mask = r.d_mask_alloc + kPadBytes;
  SG_CUDA(cudaMemsetAsync(r.d_codes_alloc, 0, tot, c->st));
  SG_CUDA(cudaMemsetAsync(r.d_mask_alloc, 0x55, tot, c->st));
  std::vector<uint8_t> hc(codes, codes + nb);
  if (n_codes & 3) hc[nb - 1] &= (uint8_t)((1u << (2 * (n_codes & 3))) - 1);  // zero past the end
  SG_CUDA(cudaMemcpyAsync(r.d_codes, hc.data(), nb, cudaMemcpyHostToDevice, c->st));
  std::vector<uint8_t> hm(nb, 0);
  if (mask) memcpy(hm.data(), mask, nb);
  for (int64_t k = n_codes; k & 3; ++k) hm[k >> 2] |= (uint8_t)(1u << ((k & 3) << 1));  // masked past the end
  SG_CUDA(cudaMemcpyAsync(r.d_mask, hm.data(), nb, cudaMemcpyHostToDevice, c->st));
  SG_CUDA(cudaMalloc(&r.d_gexp_alloc, n_codes + 2 * kGexpPad + 16));
  SG_CUDA(cudaMemsetAsync(r.d_gexp_alloc, 0, n_codes + 2 * kGexpPad + 16, c->st));
  r.d_gexp = r.d_gexp_alloc + kGexpPad;
  launch_expand_genome(r.d_codes, n_codes, r.d_gexp, c->st);
  r.rs.assign(rs, rs + std::max(n_regions, 0));
  r.re.assign(re, re + std::max(n_regions, 0));
  SG_CUDA(cudaStreamSynchronize(c->st));
  c->refs.push_back(std::move(r));
  c->indexed = false;
  return 0;
}

extern "C" int stormgpu_build_index(stormgpu_ctx* c) {
  if (!c) return STORMGPU_EINVAL;
  SG_CUDA(cudaSetDevice(c->p.device));
  SG_CUDA(cudaEventRecord(c->ev[0], c->st));
  int64_t launches = 0;
  c->indexed = false;  // until every table is there again
  for (auto& r : c->refs) {
    for (auto& ix : r.idx) {  // of the last build, from the stream-ordered pool
      if (ix.first) cudaFreeAsync(ix.first, c->st);
      if (ix.map) cudaFreeAsync(ix.map, c->st);
    }
    r.idx.assign(c->seeds.n, DevIndex());
    const int rc = build_indexes(r.d_codes, r.n, r.rs.data(), r.re.data(), (int)r.rs.size(), c->seeds.s, c->seeds.n,
                                 c->p.stdev_distance, r.idx.data(), c->st, &launches);
    if (rc) return rc;
  }
  SG_CUDA(cudaEventRecord(c->ev[1], c->st));
  SG_CUDA(cudaStreamSynchronize(c->st));
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
  c->stats.ms_index = ms;
  c->stats.kernels += launches;
  c->indexed = true;
  return 0;
}

// Candidate lists of one strand pass are bounded: a batch that would need more is mapped in
// halves (reads are independent, so the results are the same).
constexpr int64_t kMaxCandidatesPerPass = 1000000000;
constexpr int64_t kMaxPassingPerPass = 100000000;  // their tracebacks are kept until the replay
// Read streams of the banded core held at once: 1.3 KB a read of 150 codes with qualities, which a batch of
// a hundred million reads has no room for.  A larger batch is cut up front, into pieces of 3 million reads.
constexpr int64_t kMaxStreamBytes = (int64_t)4 << 30;
constexpr int kSplitBatch = 1;

// S += s (everything but the index build time)
static void add_stats(stormgpu_stats& S, const stormgpu_stats& s) {
  S.candidates += s.candidates; S.filter_passed += s.filter_passed; S.aligned += s.aligned;
  S.seed_lookups += s.seed_lookups; S.hit_positions += s.hit_positions; S.filter_cells += s.filter_cells;
  S.align_cells += s.align_cells; S.kernels += s.kernels; S.filter_band_cells += s.filter_band_cells;
  S.ms_gather += s.ms_gather; S.ms_filter += s.ms_filter; S.ms_align += s.ms_align; S.passes += s.passes;
  S.ms_replay += s.ms_replay; S.ms_total += s.ms_total; S.graph_passes += s.graph_passes;
}

// sort keys of the length order: key = read length, value = read index
static __global__ void length_keys_kernel(const int16_t* __restrict__ lengths, int64_t n, uint32_t* __restrict__ keys,
                                          uint32_t* __restrict__ vals) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    keys[i] = (uint32_t)(uint16_t)lengths[i];
    vals[i] = (uint32_t)i;
  }
}

// Work weight of a read: its seed positions, about L - 15 (candidates grow with them).
__host__ __device__ static inline int read_weight(int L) { return L > 16 ? L - 15 : 1; }

// What a call needs of its reads' lengths: the longest, 1024 less the shortest (both from 0 up, so that
// one maximum gives them), and the batch's weight.
struct LengthStats {
  unsigned long long longest, shortest_c, weight;
};

__global__ void __launch_bounds__(256) length_stats_kernel(const int16_t* __restrict__ lengths, int64_t n, LengthStats* out) {
  int hi = 0, lo_c = 0;
  unsigned long long w = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int L = lengths[i];
    hi = max(hi, L);
    lo_c = max(lo_c, STORMGPU_MAX_READ_LEN - L);
    w += (unsigned long long)read_weight(L);
  }
  hi = __reduce_max_sync(0xffffffffu, hi);
  lo_c = __reduce_max_sync(0xffffffffu, lo_c);
  for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&out->longest, (unsigned long long)hi);
    atomicMax(&out->shortest_c, (unsigned long long)lo_c);
    atomicAdd(&out->weight, w);
  }
}

// ------------------------------------------------------------------------------ passes ahead
//
// Every strand pass of a call enqueued without waiting for the device: the lists are sized up front
// (from the densest pass of the last calls, +25 %), every launch takes its list size from device
// memory, and a gate after the gather, the filter and the score bound writes the size the next stages
// take, or 0 with a status when a list would not fit (or the batch must be cut): the passes from there
// on then do nothing, and the host, reading the status once at the end, maps the call again with the
// host-synced passes.
//
// Plain launches, not a graph: a graph has to be captured again for every batch (its sizes and pointers
// are the batch's), which takes the host as long as launching, and the device waits for it; a batch of
// another size often has another number of scan launches and a new executable graph (a chain served in
// batches of 100 to 4,000 reads: 21 ms with graphs, 15 with plain launches; 400,000 reads: the same).

constexpr int kHostSynced = 2;

// Words of c->counters.  The stage counters, which passes enqueued ahead add up; what a pass starts
// with zeroed; and their state.
enum : int {
  kCntAlign = 1,   // band cells of the alignments ([2] to [6]: filter cells, index lookups, index positions,
                   // candidates, band cells of the filter)
  kCntSums = 7,
  kCntPass = 7,    // [7] candidates listed, [8] list overflow, [9..15] work cursors, [16..] those of the rounds
  kCntSelect = 24, // tickets of the two selections
  kCntBig = 26,    // int32: reads on the gather's large, huge and small lists, and above the huge slices
  kCntRounds = 28, // round_count, then int32 active_count, then the long list's count
  kGsCand = 44,    // candidates the filter of the current pass takes (0: skipped)
  kGsPass,         // passing candidates the score bound of the current pass takes (0: skipped)
  kGsKept,         // candidates the alignment of the current pass takes (0: skipped)
  kGsStatus,       // 1: a list outgrew its capacity, 2: the batch must be cut, 4: too many passing
  kGsPassed,       // sums over the passes
  kGsAligned,
  kGsMaxCand,      // densest pass
  kGsMaxPass,
  kGsMaxKept,
  kCounters = 56
};

static __global__ void gate_gather_kernel(const unsigned long long* __restrict__ counters, int64_t cand_cap,
                                          int64_t cand_max, unsigned long long* __restrict__ gs) {
  const int32_t* big_count = reinterpret_cast<const int32_t*>(counters + kCntBig);
  const unsigned long long u = counters[7];
  unsigned long long s = gs[kGsStatus];
  // candidate list overflow, a read above the slices of the last gather launch, or a full list
  if (counters[8] || big_count[3] > 0 || u > (unsigned long long)cand_cap) s |= 1;
  if (u > (unsigned long long)cand_max) s |= 2;
  gs[kGsStatus] = s;
  gs[kGsCand] = s ? 0 : u;
  if (u > gs[kGsMaxCand]) gs[kGsMaxCand] = u;
}

static void set_densities(stormgpu_ctx* c, double cand, double pass, double kept) {
  c->dens_cand = cand;
  c->dens_pass = pass;
  c->gdens_cand = std::max(cand, 0.9 * c->gdens_cand);
  c->gdens_pass = std::max(pass, 0.9 * c->gdens_pass);
  c->gdens_kept = std::max(kept, 0.9 * c->gdens_kept);
}

// What the passes of one call share (set up by map_device_once before them).
constexpr int kRoundCounts = kMaxAlignRounds + 1;

struct PassSetup {
  ScoreParams sp;
  ReadsDev fwd, rev;
  int64_t n;
  int maxL, minL;
  double wsum;
  int wpr;          // scratch words per row of an alignment
  int64_t tbs;      // traceback bytes per aligned candidate
  int rounds;       // alignment rounds
  int filter_H;     // band registers of the filter's core, 0: the core of filter_core.cuh
  int bound_H;      // band registers of the score bound, 0: every passing candidate is aligned
  stormgpu_results* out;
};

// Read streams of one pass for the filter, and for the score bound too when its band is the same.
static void launch_filter_streams(stormgpu_ctx* c, const PassSetup& P, const ReadsDev& rd, cudaStream_t st) {
  if (!P.filter_H) {
    launch_expand_reads(rd, c->rexp.p, rexp_stride(P.maxL), st);
    return;
  }
  const bool both = P.filter_H == P.bound_H;
  launch_band_streams(rd, P.filter_H, band_stream_words(P.maxL, P.filter_H), c->bstream.p,
                      both && rd.levels ? c->wstream.p : nullptr, c->bound_c, st);
}

static void set_filter_job(stormgpu_ctx* c, const PassSetup& P, const ReadsDev& rd, const RefSeq& R, FilterJob& job) {
  const ScoreParams& sp = P.sp;
  job.rows = c->tune.filter_rows;
  job.fr = c->fr.p; job.fd = c->fd.p; job.flag = c->flag.p; job.codes = rd.codes;
  job.cstride = rd.cstride; job.lengths = rd.lengths; job.genome = R.d_codes; job.W = sp.W; job.Is = sp.Is;
  job.fm = sp.fm; job.fx = sp.fx; job.fo = sp.fo; job.fe = sp.fe; job.fthr = sp.fthr;
  job.counters = c->counters.p;
  job.gexp = R.d_gexp; job.rexp = c->rexp.p; job.rstride = rexp_stride(P.maxL); job.min_len = P.minL;
  job.band_H = P.filter_H; job.band = c->filter_c; job.bs = c->bstream.p;
  job.bwords = P.filter_H ? band_stream_words(P.maxL, P.filter_H) : 0;
}

// The score bound of one pass: streams of its reads (unless the filter's serve), then the flags of the
// passing candidates (q_read, q_diag), their number read from n_dev when given.
static void launch_bound_pass(stormgpu_ctx* c, const PassSetup& P, const ReadsDev& rd, const RefSeq& R, int64_t n,
                              const int64_t* n_dev, cudaStream_t st) {
  const int64_t words = band_stream_words(P.maxL, P.bound_H);
  if (P.filter_H != P.bound_H)
    launch_band_streams(rd, P.bound_H, words, c->bstream.p, rd.levels ? c->wstream.p : nullptr, c->bound_c, st);
  BoundJob job;
  memset(&job, 0, sizeof(job));
  job.n = n; job.n_dev = n_dev; job.read = c->q_read.p; job.diag = c->q_diag.p; job.lengths = rd.lengths;
  job.gexp = R.d_gexp; job.rs = c->bstream.p; job.ws = rd.levels ? c->wstream.p : nullptr; job.words = words;
  job.H = P.bound_H; job.I = P.sp.I; job.Is = P.sp.Is; job.min_score = P.sp.min_score;
  job.match = P.sp.pair[0][3]; job.mismatch = -P.sp.pair[1][3];
  job.flag = c->flag.p; job.ub = c->q_ub.p;
  launch_score_bound(job, c->bound_c, st);
}

// Buffers of the replay's lists: two lists of active reads, and with rounds the round's slots.
static int round_lists_grow(stormgpu_ctx* c, int64_t n, int64_t kept, int rounds) {
  if (c->active.grow(2 * n) || c->long_list.grow(n)) return STORMGPU_ENOMEM;
  if (rounds > 1 && (c->thr.grow(n) || c->round_cur.grow(2 * n) || c->round_slots.grow(kept))) return STORMGPU_ENOMEM;
  return 0;
}

// Their pointers for round k.
static void round_buffers(stormgpu_ctx* c, int k, PassBuffers& pb) {
  const int64_t half = c->active.cap / 2;
  pb.round = k;
  pb.round_count = c->counters.p + kCntRounds + k;  // zeroed with the counters of the pass
  pb.active = c->active.p + (k & 1 ? half : 0);
  pb.active_next = c->active.p + (k & 1 ? 0 : half);
  pb.active_count = reinterpret_cast<int32_t*>(c->counters.p + kCntRounds + kRoundCounts) + k;
  pb.cursor = c->counters.p + 16 + k;
}

static void setup_rounds(stormgpu_ctx* c, int rounds, PassBuffers& pb) {
  round_buffers(c, 0, pb);
  if (rounds > 1) {
    pb.round_slots = c->round_slots.p;
    pb.round_cur = c->round_cur.p;
    pb.thr = c->thr.p;
  }
}

static KeptList kept_list(stormgpu_ctx* c, const PassSetup& P, int64_t n, const int64_t* n_dev) {
  KeptList kl;
  kl.n = n;
  kl.n_dev = n_dev;
  kl.diag = c->k_diag.p;
  kl.ub = P.bound_H ? c->k_ub.p : nullptr;
  kl.long_list = c->long_list.p;
  kl.long_count = reinterpret_cast<int32_t*>(c->counters.p + kCntRounds + 2 * kRoundCounts);
  kl.sort_cap = c->tune.gather_warp_cap;  // more come from the block gather, in order
  return kl;
}

static int32_t* big_count(stormgpu_ctx* c) { return reinterpret_cast<int32_t*>(c->counters.p + kCntBig); }

// The lists of reads the warp gather hands on: at most kSmallGatherCap positions, more, and too many for
// shared memory.  Their cursors are zeroed with the counters of the pass.
static GatherList small_gather_list(stormgpu_ctx* c, int64_t n, const int32_t* n_dev) {
  return {c->small_list.p, c->small_h.p, n, n_dev, c->counters.p + 9, c->huge_list.p, c->huge_h.p, big_count(c) + 1};
}
static GatherList large_gather_list(stormgpu_ctx* c, int64_t n, const int32_t* n_dev) {
  return {c->big_list.p, c->big_h.p, n, n_dev, c->counters.p + 14, c->huge_list.p, c->huge_h.p, big_count(c) + 1};
}
static GatherList huge_gather_list(stormgpu_ctx* c, int64_t reads, int64_t n, const int32_t* n_dev) {
  return {c->huge_list.p, c->huge_h.p, n, n_dev, c->counters.p + 15, c->huge_list.p + reads, c->huge_h.p + reads,
          big_count(c) + 1};
}

// List capacities of a call whose passes are enqueued ahead.
struct AheadCaps {
  int64_t cand, pass, kept;
  int64_t grid_h;  // blocks of the gather for the reads with the most positions
};

// The lists such a call needs (false: they could not be allocated, and the call runs host-synced).
static bool ahead_buffers(stormgpu_ctx* c, const PassSetup& P, AheadCaps* caps) {
  const int64_t n = P.n;
  const int64_t want_cand = (int64_t)(c->gdens_cand * P.wsum * 1.25) + 61440;  // small calls: one scan block
  const int64_t spare = std::min<int64_t>(4096, 64 * n);  // few reads: few enough for the wave alignment alone
  const int64_t want_pass = (int64_t)(c->gdens_pass * P.wsum * 1.25) + spare;
  const int64_t want_kept = P.bound_H ? (int64_t)(c->gdens_kept * P.wsum * 1.25) + spare : want_pass;
  caps->grid_h = std::max<int64_t>(1, std::min<int64_t>(gather_huge_grid(), ((int64_t)1 << 25) / c->huge_cap));
  if (c->fr.grow(want_cand) || c->fd.grow(want_cand) ||
      c->big_tmp.grow(caps->grid_h * c->huge_cap))
    return false;
  if (P.bound_H && (c->q_read.grow(want_pass) || c->q_diag.grow(want_pass) || c->q_ub.grow(want_pass) ||
                    c->k_ub.grow(want_kept) || c->p_ub.grow(want_kept)))
    return false;
  if (c->p_read.grow(want_kept) || c->p_diag.grow(want_kept) || c->k_diag.grow(want_kept) || c->a_score.grow(want_kept) ||
      c->a_bound.grow(want_kept) || c->a_tblen.grow(want_kept) || c->a_pos.grow(want_kept * 4) ||
      c->a_tb.grow(want_kept * P.tbs))
    return false;
  // what was asked for, not what a buffer has grown to: the grids are sized by it
  caps->cand = want_cand;
  caps->kept = want_kept;
  caps->pass = P.bound_H ? want_pass : caps->kept;
  const int64_t longest = std::max(caps->cand, caps->pass);
  if (c->flag.grow(longest) || c->foff.grow(select_tiles(longest) + 1)) return false;
  if ((P.rounds > 1 || caps->kept > wave_slots(P.sp)) &&
      c->scratch.grow(align_workers(caps->kept, P.sp) * (int64_t)P.maxL * P.wpr))
    return false;
  return round_lists_grow(c, n, caps->kept, P.rounds) == 0;
}

// The launches of every pass on c's stream, each list size read from the device; nothing here waits for
// the device.  E: the stage events, per_pass per pass.
static int enqueue_passes(stormgpu_ctx* c, const PassSetup& P, const AheadCaps& caps, int per_pass,
                                int64_t& launches) {
  cudaStream_t st = c->st;
  const int64_t cand_cap = caps.cand, pass_cap = caps.pass, kept_cap = caps.kept, grid_h = caps.grid_h;
  const ScoreParams& sp = P.sp;
  const int64_t n = P.n;
  unsigned long long* gs = c->counters.p;
  const int rounds = P.rounds;
  auto rec = [&](cudaEvent_t e) { return cudaEventRecord(e, st); };
  SG_CUDA(cudaMemsetAsync(gs, 0, sizeof(unsigned long long) * kCounters, st));
  int pi = 0;
  for (size_t ref_id = 0; ref_id < c->refs.size(); ++ref_id) {
    RefSeq& R = c->refs[ref_id];
    IndexView ix;
    memset(&ix, 0, sizeof(ix));
    for (int si = 0; si < c->seeds.n; ++si) { ix.first[si] = R.idx[si].first; ix.map[si] = R.idx[si].map; }
    for (int strand = 0; strand < 2; ++strand) {
      if (!(c->p.senses & (1 << strand))) continue;
      const ReadsDev& rd = strand ? P.rev : P.fwd;
      cudaEvent_t* E = c->gev.data() + (size_t)pi * per_pass;
      ++pi;
      SG_CUDA(rec(E[0]));
      // hit gather: the warp kernel, then the block kernels over the lists it filled, then the
      // reads above the block kernel's slices (reads above this launch's slices end the
      // call: the host-synced passes size their slices to fit)
      if (pi > 1)
        SG_CUDA(cudaMemsetAsync(c->counters.p + kCntPass, 0, sizeof(unsigned long long) * (kGsCand - kCntPass), st));
      GatherOut go;
      go.fr = c->fr.p; go.fd = c->fd.p; go.cap = cand_cap; go.counters = c->counters.p;
      go.big_list = c->big_list.p; go.big_h = c->big_h.p; go.small_list = c->small_list.p;
      go.small_h = c->small_h.p; go.big_count = big_count(c);
      go.cursor = c->counters.p + 12;
      go.reads_per_steal = c->tune.gather_reads_per_steal;
      go.warp_cap = c->tune.gather_warp_cap;
      launch_gather_fused(rd, ix, sp.I, go, c->seeds, st);
      launch_gather_sort(rd, ix, sp.I, R.n, small_gather_list(c, n, big_count(c) + 2), true, go, c->seeds, st);
      launch_gather_sort(rd, ix, sp.I, R.n, large_gather_list(c, n, big_count(c) + 0), false, go, c->seeds, st);
      GatherList hl = huge_gather_list(c, n, n, big_count(c) + 1);
      hl.above_count = big_count(c) + 3;
      launch_gather_huge(rd, ix, sp.I, R.n, hl, c->big_tmp.p, (int)c->huge_cap, grid_h, go, c->seeds, st);
      gate_gather_kernel<<<1, 1, 0, st>>>(c->counters.p, cand_cap, kMaxCandidatesPerPass, gs);
      launches += 5;
      SG_CUDA(rec(E[1]));
      // filter over the gate's candidate count
      FilterJob job;
      memset(&job, 0, sizeof(job));
      if (c->tune.filter_cursor) job.cursor = c->counters.p + 10;
      job.n = cand_cap; job.n_dev = gs + kGsCand;
      set_filter_job(c, P, rd, R, job);
      launch_filter_streams(c, P, rd, st);
      launch_filter_flat_job(job, sp, filter_dpx_ok(sp, P.maxL), st);
      launches += 2;
      SG_CUDA(rec(E[2]));
      // the passing candidates, in order
      const SelectGate passing{gs + kGsStatus, gs + kGsPass, gs + kGsPassed, gs + kGsMaxPass, pass_cap,
                               n > 1 ? kMaxPassingPerPass : INT64_MAX};
      const SelectGate kept{gs + kGsStatus, gs + kGsKept, gs + kGsAligned, gs + kGsMaxKept, kept_cap, INT64_MAX};
      auto select = [&](int64_t cap, int take, int which, const SelectGate& g0, const SelectGate& g1, const int32_t* fr,
                        const int32_t* fd, int32_t* o_read, int32_t* o_diag, int64_t ocap, const int16_t* ub, int16_t* o_ub) {
        if (cand_cap <= kSelectSmall) {
          launch_select_small(cap, gs + take, c->flag.p, g0, g1, fr, fd, o_read, o_diag, ocap, ub, o_ub, st);
          launches++;
          return;
        }
        launch_select_count(cap, gs + take, c->flag.p, c->foff.p, gs + kCntSelect + which, g0, g1, st);
        launch_select_write(cap, gs + take, c->flag.p, c->foff.p, fr, fd, o_read, o_diag, ocap, ub, o_ub, st);
        launches += 2;
      };
      PassBuffers pb;
      memset(&pb, 0, sizeof(pb));
      pb.pstart = c->pstart.p; pb.pcount = c->pcount.p;
      pb.p_read = c->p_read.p; pb.p_diag = c->p_diag.p;
      if (P.bound_H) {
        // the candidates whose score can exceed -t, in order
        select(cand_cap, kGsCand, 0, passing, {}, c->fr.p, c->fd.p, c->q_read.p, c->q_diag.p, pass_cap, nullptr, nullptr);
        launch_bound_pass(c, P, rd, R, pass_cap, reinterpret_cast<const int64_t*>(gs + kGsPass), st);
        select(pass_cap, kGsPass, 1, kept, {}, c->q_read.p, c->q_diag.p, c->p_read.p, c->k_diag.p, kept_cap, c->q_ub.p,
               c->k_ub.p);
        pb.ub = c->p_ub.p;
        launches++;
      } else {
        select(cand_cap, kGsCand, 0, passing, kept, c->fr.p, c->fd.p, c->p_read.p, c->k_diag.p, kept_cap, nullptr, nullptr);
      }
      const int64_t* np = reinterpret_cast<const int64_t*>(gs + kGsKept);
      setup_rounds(c, rounds, pb);
      launch_slot_lists(kept_list(c, P, kept_cap, np), c->p_ub.p, pb, align_round_take(0, rounds), st);
      launches += kept_cap <= kSlotsSmall ? 1 : 3;
      pb.a_score = c->a_score.p; pb.a_bound = c->a_bound.p; pb.a_tblen = c->a_tblen.p;
      pb.a_pos = c->a_pos.p; pb.a_tb = c->a_tb.p; pb.tbs = P.tbs;
      pb.npass_dev = np;
      pb.steal = c->tune.align_steal;
      pb.a_scratch = c->scratch.p;
      pb.cells = c->counters.p + kCntAlign;
      if (rounds == 1) {
        pb.wave = wave_slots(sp);
        if (pb.wave) launch_align_wave(rd, sp, R.d_codes, R.d_mask, 0, kept_cap, pb, P.maxL, st);
        if (kept_cap > pb.wave) launch_align(rd, sp, R.d_codes, R.d_mask, 0, kept_cap, pb, st);
        launches += (pb.wave > 0) + (kept_cap > pb.wave);
        SG_CUDA(rec(E[3]));
        launch_replay(n, sp, (int)ref_id, strand ? -1 : 1, pb, 0, P.out->hits, P.out->tb, P.out->tb_stride,
                      P.out->mapped, st);
        launches++;
      } else {
        SG_CUDA(rec(E[5]));
        for (int k = 0; k < rounds; ++k) {
          round_buffers(c, k, pb);
          launch_align(rd, sp, R.d_codes, R.d_mask, 0, kept_cap, pb, st);
          SG_CUDA(rec(E[6 + 2 * k]));
          launch_replay(n, sp, (int)ref_id, strand ? -1 : 1, pb, align_round_take(k + 1, rounds), P.out->hits,
                        P.out->tb, P.out->tb_stride, P.out->mapped, st);
          SG_CUDA(rec(E[7 + 2 * k]));
          launches += 2;
        }
        SG_CUDA(rec(E[3]));
      }
      SG_CUDA(rec(E[4]));
    }
  }
  return 0;
}

// Every pass of the call enqueued ahead.  0: done (results in P.out, stats in c->stats); kHostSynced: the
// results are not usable (a list did not fit) and the call must run the host-synced passes; else an
// error code.
static int map_passes_ahead(stormgpu_ctx* c, const PassSetup& P, int64_t launches) {
  cudaStream_t st = c->st;
  AheadCaps caps;
  if (!ahead_buffers(c, P, &caps)) {
    cudaGetLastError();
    c->work.over = false;  // the host-synced passes allocate what they need, no more
    return kHostSynced;
  }
  const int rounds = P.rounds;
  const int per_pass = 5 + (rounds > 1 ? 1 + 2 * rounds : 0);
  int npasses = 0;
  for (size_t r = 0; r < c->refs.size(); ++r)
    for (int strand = 0; strand < 2; ++strand) npasses += (c->p.senses >> strand) & 1;
  while (c->gev.size() < (size_t)npasses * per_pass) {
    cudaEvent_t e;
    SG_CUDA(cudaEventCreate(&e));
    c->gev.push_back(e);
  }
  unsigned long long h[kCounters];
  SG_CUDA(cudaEventRecord(c->ev[6], st));
  if (const int e = enqueue_passes(c, P, caps, per_pass, launches)) return e;
  SG_CUDA(cudaEventRecord(c->ev[7], st));
  SG_CUDA(cudaMemcpyAsync(h, c->counters.p, sizeof(h), cudaMemcpyDeviceToHost, st));
  SG_CUDA(cudaStreamSynchronize(st));
  SG_CUDA(cudaGetLastError());
  if (h[kGsStatus]) return kHostSynced;
  stormgpu_stats& S = c->stats;
  S.candidates = (int64_t)h[5];
  S.filter_cells = (int64_t)h[2];
  S.filter_band_cells = (int64_t)h[6];
  S.seed_lookups = (int64_t)h[3];
  S.hit_positions = (int64_t)h[4];
  S.filter_passed = (int64_t)h[kGsPassed];
  S.aligned = (int64_t)h[kGsAligned];
  S.align_cells = (int64_t)h[kCntAlign];
  S.passes = npasses;
  S.graph_passes = npasses;
  // stage times (as the host-synced passes split them)
  float tg = 0, tf = 0, ta = 0, tr = 0, tt = 0;
  for (int pi = 0; pi < npasses; ++pi) {
    const cudaEvent_t* E = c->gev.data() + (size_t)pi * per_pass;
    float a = 0, b = 0, d = 0, e = 0;
    cudaEventElapsedTime(&a, E[0], E[1]);
    cudaEventElapsedTime(&b, E[1], E[2]);
    cudaEventElapsedTime(&d, E[2], E[3]);
    cudaEventElapsedTime(&e, E[3], E[4]);
    for (int k = 0; rounds > 1 && k < rounds; ++k) {  // the rounds' replays count as replay time
      float x = 0;
      cudaEventElapsedTime(&x, E[6 + 2 * k], E[7 + 2 * k]);
      d -= x;
      e += x;
    }
    tg += a; tf += b; ta += d; tr += e;
  }
  cudaEventElapsedTime(&tt, c->ev[6], c->ev[7]);
  cudaGetLastError();
  S.ms_gather = tg; S.ms_filter = tf; S.ms_align = ta; S.ms_replay = tr; S.ms_total = tt;
  S.kernels = launches;
  if (P.wsum > 0) set_densities(c, (double)h[kGsMaxCand] / P.wsum, (double)h[kGsMaxPass] / P.wsum, (double)h[kGsMaxKept] / P.wsum);
  return 0;
}

// Alignment rounds of a pass that aligns about `kept` candidates of n reads, at most `most`.  Rounds pay
// where reads have so many candidates that each round lets the bound drop most of what is left: mixed
// reads of a repeat-rich genome at -i 15, 360 per read and strand, alignment 17.1 -> 13.1 ms with 4 rounds
// (43 % of the cells).  With few per read all the rounds do is to align them a part at a time, each
// taking as long as its longest read: 14 per read 4.8 -> 9.6 ms (ragged reads at -i 5), 1.6 per read
// 0.61 -> 0.86 ms (48 Mbp), as in a call of a few reads.
static int align_rounds(int most, int64_t n, double kept) { return n <= 256 || kept < 32.0 * (double)n ? 1 : most; }

// The lengths' measures: from the host's copy when there is one, else by a kernel (400,000 lengths copied
// and walked by the host took 1 ms of a 31 ms call).
static int length_stats(stormgpu_ctx* c, const stormgpu_reads* reads, const int16_t* lengths, LengthStats* out) {
  memset(out, 0, sizeof(*out));
  const int64_t n = reads->n;
  if (n <= 0) return 0;
  if (lengths) {
    int hi = 0, lo_c = 0;
    int64_t w = 0;
    for (int64_t r = 0; r < n; ++r) {
      const int L = lengths[r];
      hi = std::max(hi, L);
      lo_c = std::max(lo_c, STORMGPU_MAX_READ_LEN - L);
      w += read_weight(L);
    }
    *out = {(unsigned long long)hi, (unsigned long long)lo_c, (unsigned long long)w};
    return 0;
  }
  if (c->counters.grow(kCounters)) return STORMGPU_ENOMEM;
  LengthStats* d = reinterpret_cast<LengthStats*>(c->counters.p);
  SG_CUDA(cudaMemsetAsync(d, 0, sizeof(*d), c->st));
  length_stats_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 4), 256, 0, c->st>>>(reads->lengths, n, d);
  SG_CUDA(cudaMemcpyAsync(out, d, sizeof(*d), cudaMemcpyDeviceToHost, c->st));
  SG_CUDA(cudaStreamSynchronize(c->st));
  return 0;
}

// Band registers of the banded core for the filter and for the score bound (nucleotide space, a band it is
// instantiated for), 0 where it is not used.
struct BandWidths {
  int filter, bound;
  // bytes of the read streams of n reads, the longest of max_len
  int64_t stream_bytes(int64_t n, int max_len, bool levels) const {
    const int64_t words = std::max(filter ? band_stream_words(max_len, filter) : 0, bound ? band_stream_words(max_len, bound) : 0);
    return n * words * (int64_t)sizeof(uint32_t) * (bound && levels ? 2 : 1);
  }
};

static BandWidths band_widths(stormgpu_ctx* c, const ScoreParams& sp) {
  if (!c->band_set) {
    c->filter_c = band_filter_consts(sp.fm, sp.fx, sp.fo, sp.fe, sp.fthr);
    memset(&c->bound_c, 0, sizeof(c->bound_c));
    if (!sp.colour && sp.I <= kMaxBoundIndels) c->bound_c = band_bound_consts(sp.pair, sp.gap_open, sp.gap_ext);
    c->band_set = true;
  }
  return {filter_band_registers(sp.W, c->filter_c), c->bound_c.ok ? bound_registers(sp.I) : 0};
}

static int map_device_once(stormgpu_ctx* c, const stormgpu_reads* reads, const LengthStats& ls, stormgpu_results* out) {
  if (!c->indexed) { sg_set_error("stormgpu_build_index must be called before mapping"); return STORMGPU_ESTATE; }
  cudaStream_t st = c->st;
  const int64_t n = reads->n;
  const ScoreParams sp = make_score_params(c->p);
  stormgpu_stats& S = c->stats;
  double ms_index = S.ms_index;
  memset(&S, 0, sizeof(S));
  S.ms_index = ms_index;
  int64_t launches = 0;
  const int maxL = (int)ls.longest, minL = STORMGPU_MAX_READ_LEN - (int)ls.shortest_c;
  const double wsum = (double)ls.weight;  // the batch's work weight (read_weight)
  if (maxL > STORMGPU_MAX_READ_LEN) { sg_set_error("read longer than %d", STORMGPU_MAX_READ_LEN); return STORMGPU_EINVAL; }
  if (out->tb_stride < (maxL + c->p.allowed_indels + 1) / 2) { sg_set_error("tb_stride too small"); return STORMGPU_EINVAL; }
  launch_init_results(n, out->hits, out->mapped, out->tb, out->tb_stride, st);
  launches++;
  if (n == 0) return 0;
  ReadsDev fwd{n, reads->codes, reads->code_stride, reads->levels, reads->level_stride, reads->lengths, nullptr};
  if (minL != maxL) {
    // reads of several lengths: the gather visits them grouped by length (a stable sort of the
    // read indices by length); a batch in any read order then runs like one sorted by length
    if (c->ord.grow(4 * n) || c->ord_tmp.grow(radix_tmp_bytes(n) / 4 + 16)) return STORMGPU_ENOMEM;
    uint32_t *k0 = c->ord.p, *v0 = k0 + n, *k1 = v0 + n, *v1 = k1 + n;
    length_keys_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, st>>>(reads->lengths, n, k0, v0);
    int bits = 1;
    while ((1 << bits) <= maxL) ++bits;
    const int which = radix_sort_pairs(k0, v0, k1, v1, n, bits, c->ord_tmp.p, st);
    fwd.order = reinterpret_cast<const int32_t*>(which ? v1 : v0);
    launches += 1 + 3 * ((bits + kRadixBits - 1) / kRadixBits);
  }
  ReadsDev rev = fwd;
  if (c->p.senses & 2) {
    if (c->rcodes.grow(n * reads->code_stride)) return STORMGPU_ENOMEM;
    if (reads->levels && c->rlevels.grow(n * reads->level_stride)) return STORMGPU_ENOMEM;
    launch_reverse_reads(fwd, c->p.colour ? reads->first_levels : nullptr, c->p.colour, c->rcodes.p,
                         reads->levels ? c->rlevels.p : nullptr, st);
    launches++;
    rev.codes = c->rcodes.p;
    rev.levels = reads->levels ? c->rlevels.p : nullptr;
  }
  if (c->pstart.grow(n) || c->pcount.grow(n) ||
      c->big_list.grow(n) || c->big_h.grow(n) || c->small_list.grow(n) || c->small_h.grow(n) ||
      c->huge_list.grow(2 * n) || c->huge_h.grow(2 * n) || c->counters.grow(kCounters) ||
      c->fr.grow(std::max<int64_t>(n * 64, 1 << 20)) ||
      c->fd.grow(std::max<int64_t>(n * 64, 1 << 20)))
    return STORMGPU_ENOMEM;
  const int BW = 2 * sp.I + 1;
  const int wpr = (2 * BW + 31) / 32 + (sp.colour ? (BW + 31) / 32 : 0);
  const int64_t tbs = ((maxL + sp.I + 1) / 2 + 7) & ~7LL;
  const BandWidths bw = band_widths(c, sp);
  const int filter_H = bw.filter, bound_H = bw.bound;
  {
    const int64_t words = n * std::max(filter_H ? band_stream_words(maxL, filter_H) : 0,
                                       bound_H ? band_stream_words(maxL, bound_H) : 0);
    if (c->bstream.grow(words) || (bound_H && reads->levels && c->wstream.grow(words)) ||
        (!filter_H && c->rexp.grow(n * rexp_stride(maxL))))
      return STORMGPU_ENOMEM;
  }
  // rounds drop candidates by their bound: none in a batch whose reads, at their mean length, are too long
  // for a bound above -t (1,000 reads of 400 codes at -i 15, 102 candidates per read and strand: the call
  // 8.7 ms with 4 rounds, 3.7 with one)
  const int mean_len = (int)(wsum / (double)n) + 15;
  const bool has_bound = bound_H && band_bound_limit(sp.pair[0][3], -sp.pair[1][3], mean_len) > sp.min_score;
  const int most_rounds = !has_bound ? 1 : std::max(1, std::min<int>(c->tune.align_rounds, kMaxAlignRounds));
  const int rounds_ahead = align_rounds(most_rounds, n, c->gdens_kept * wsum);
  const PassSetup P{sp, fwd, rev, n, maxL, minL, wsum, wpr, tbs, rounds_ahead, filter_H, bound_H, out};
  if (c->graphs && c->gdens_cand > 0 && c->huge_cap <= ((int64_t)1 << 22)) {
    const int g = map_passes_ahead(c, P, launches);
    if (g != kHostSynced) return g;
    // a list outgrew its capacity: the passes again, each sized by the host (the replays of the
    // first passes may have updated the results)
    launch_init_results(n, out->hits, out->mapped, out->tb, out->tb_stride, st);
    launches++;
  }
  float tg = 0, tf = 0, ta = 0, tr = 0;
  int64_t max_cand = 0, max_pass = 0, max_kept = 0;  // densest strand pass of this call
  SG_CUDA(cudaEventRecord(c->ev[6], st));
  for (size_t ref_id = 0; ref_id < c->refs.size(); ++ref_id) {
    RefSeq& R = c->refs[ref_id];
    IndexView ix;
    memset(&ix, 0, sizeof(ix));
    for (int si = 0; si < c->seeds.n; ++si) { ix.first[si] = R.idx[si].first; ix.map[si] = R.idx[si].map; }
    for (int strand = 0; strand < 2; ++strand) {
      if (!(c->p.senses & (1 << strand))) continue;
      const ReadsDev& rd = strand ? rev : fwd;
      int64_t utot = 0;
      SG_CUDA(cudaEventRecord(c->ev[0], st));
      for (int attempt = 0;; ++attempt) {
        // fused hit gather: sorted, de-duplicated diagonals of every read, appended to the flat
        // candidate list (fr, fd); reads with many index positions go to the block kernel
        SG_CUDA(cudaMemsetAsync(c->counters.p, 0, sizeof(unsigned long long) * kCounters, st));
        GatherOut go;
        // (a call that ran out of memory between the two leaves them of different lengths)
        go.fr = c->fr.p; go.fd = c->fd.p; go.cap = std::min(c->fr.cap, c->fd.cap); go.counters = c->counters.p;
        go.big_list = c->big_list.p; go.big_h = c->big_h.p; go.small_list = c->small_list.p;
        go.small_h = c->small_h.p; go.big_count = big_count(c);
        go.cursor = c->counters.p + 12;  // zeroed just above
        go.reads_per_steal = c->tune.gather_reads_per_steal;
        go.warp_cap = c->tune.gather_warp_cap;
        launch_gather_fused(rd, ix, sp.I, go, c->seeds, st);
        launches++;
        int32_t nbig[3] = {0, 0, 0};  // handed to the block gather with many positions, above its slice, with few
        SG_CUDA(cudaMemcpyAsync(nbig, big_count(c), sizeof(nbig), cudaMemcpyDeviceToHost, st));
        SG_CUDA(cudaStreamSynchronize(st));
        if (nbig[2] > 0) {  // reads with few positions: sorted in shared memory
          launch_gather_sort(rd, ix, sp.I, R.n, small_gather_list(c, nbig[2], nullptr), true, go, c->seeds, st);
          launches++;
        }
        if (nbig[0] > 0) {  // reads with many positions: a block with most of an SM's shared memory
          launch_gather_sort(rd, ix, sp.I, R.n, large_gather_list(c, nbig[0], nullptr), false, go, c->seeds, st);
          launches++;
          SG_CUDA(cudaMemcpyAsync(nbig + 1, big_count(c) + 1, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
          SG_CUDA(cudaStreamSynchronize(st));
          if (nbig[1] > 0) {  // beyond it: slices of the largest read's size in global memory
            std::vector<int32_t> hh(nbig[1]);
            SG_CUDA(cudaMemcpyAsync(hh.data(), c->huge_h.p, sizeof(int32_t) * nbig[1], cudaMemcpyDeviceToHost, st));
            SG_CUDA(cudaStreamSynchronize(st));
            int64_t cap2 = 65536;
            for (int k = 0; k < nbig[1]; ++k) while (cap2 < hh[k]) cap2 <<= 1;
            if (cap2 > (int64_t)1 << 30) { sg_set_error("a read has %lld index positions", (long long)cap2); return STORMGPU_EINVAL; }
            c->huge_cap = std::max<int64_t>(c->huge_cap, cap2);
            // at most 1 GiB of slices
            const int64_t grid2 = std::max<int64_t>(1, std::min<int64_t>({(int64_t)nbig[1], gather_huge_grid(),
                                                                           ((int64_t)1 << 28) / cap2}));
            if (c->big_tmp.grow(grid2 * cap2)) return STORMGPU_ENOMEM;
            launch_gather_huge(rd, ix, sp.I, R.n, huge_gather_list(c, n, nbig[1], nullptr), c->big_tmp.p, (int)cap2, grid2,
                               go, c->seeds, st);
            launches++;
          }
        }
        unsigned long long g[9];
        SG_CUDA(cudaMemcpyAsync(g, c->counters.p, sizeof(g), cudaMemcpyDeviceToHost, st));
        SG_CUDA(cudaStreamSynchronize(st));
        utot = (int64_t)g[7];
        max_cand = std::max(max_cand, utot);
        if (utot > kMaxCandidatesPerPass) return kSplitBatch;
        if (!g[8]) break;
        if (attempt > 2) { sg_set_error("internal: candidate list overflow"); return STORMGPU_EINVAL; }
        if (c->fr.grow(utot + utot / 4 + 1024) || c->fd.grow(utot + utot / 4 + 1024)) return STORMGPU_ENOMEM;
      }
      const int64_t tiles = select_tiles(utot);
      if (c->flag.grow(std::max<int64_t>(utot, 1)) || c->foff.grow(tiles + 1)) return STORMGPU_ENOMEM;
      SG_CUDA(cudaEventRecord(c->ev[1], st));
      FilterJob job;
      memset(&job, 0, sizeof(job));
      if (c->tune.filter_cursor) job.cursor = c->counters.p + 10;  // zeroed with the counters of the pass
      job.n = utot;
      set_filter_job(c, P, rd, R, job);
      launch_filter_streams(c, P, rd, st);
      launch_filter_flat_job(job, sp, filter_dpx_ok(sp, maxL), st);
      launches += 2;
      S.passes++;
      SG_CUDA(cudaEventRecord(c->ev[2], st));
      launch_select_count(utot, nullptr, c->flag.p, c->foff.p, c->counters.p + kCntSelect, {}, {}, st);
      launches++;
      unsigned long long cnt[8];
      int64_t npass = 0;
      SG_CUDA(cudaMemcpyAsync(&npass, c->foff.p + tiles, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
      SG_CUDA(cudaMemcpyAsync(cnt, c->counters.p, sizeof(cnt), cudaMemcpyDeviceToHost, st));
      SG_CUDA(cudaStreamSynchronize(st));
      S.candidates += (int64_t)cnt[5];
      S.filter_cells += (int64_t)cnt[2];
      S.filter_band_cells += (int64_t)cnt[6];
      S.seed_lookups += (int64_t)cnt[3];
      S.hit_positions += (int64_t)cnt[4];
      S.filter_passed += npass;
      max_pass = std::max(max_pass, npass);
      if (npass > kMaxPassingPerPass && n > 1) return kSplitBatch;
      PassBuffers pb;
      memset(&pb, 0, sizeof(pb));
      pb.pstart = c->pstart.p; pb.pcount = c->pcount.p;
      int64_t nkept = npass;  // candidates that are aligned
      if (npass > 0 && bound_H) {
        // those whose score can exceed -t, in order
        if (c->q_read.grow(npass) || c->q_diag.grow(npass) || c->q_ub.grow(npass)) return STORMGPU_ENOMEM;
        launch_select_write(utot, nullptr, c->flag.p, c->foff.p, c->fr.p, c->fd.p, c->q_read.p, c->q_diag.p,
                            c->q_read.cap, nullptr, nullptr, st);
        launch_bound_pass(c, P, rd, R, npass, nullptr, st);
        launch_select_count(npass, nullptr, c->flag.p, c->foff.p, c->counters.p + kCntSelect + 1, {}, {}, st);
        launches += 4;
        SG_CUDA(cudaMemcpyAsync(&nkept, c->foff.p + select_tiles(npass), sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        SG_CUDA(cudaStreamSynchronize(st));
      }
      max_kept = std::max(max_kept, nkept);
      const int rounds = align_rounds(most_rounds, n, (double)nkept);
      if (nkept > 0) {
        if (c->p_read.grow(nkept) || c->p_diag.grow(nkept) || c->k_diag.grow(nkept) || c->a_score.grow(nkept) || c->a_bound.grow(nkept) ||
            c->a_tblen.grow(nkept) || c->a_pos.grow(nkept * 4) || c->a_tb.grow(nkept * tbs) ||
            (bound_H && (c->k_ub.grow(nkept) || c->p_ub.grow(nkept))))
          return STORMGPU_ENOMEM;
        pb.p_read = c->p_read.p; pb.p_diag = c->p_diag.p;
        if (bound_H) {
          launch_select_write(npass, nullptr, c->flag.p, c->foff.p, c->q_read.p, c->q_diag.p, c->p_read.p, c->k_diag.p,
                              nkept, c->q_ub.p, c->k_ub.p, st);
          pb.ub = c->p_ub.p;
        } else {
          launch_select_write(utot, nullptr, c->flag.p, c->foff.p, c->fr.p, c->fd.p, c->p_read.p, c->k_diag.p, nkept,
                              nullptr, nullptr, st);
        }
        if (round_lists_grow(c, n, nkept, rounds)) return STORMGPU_ENOMEM;
        setup_rounds(c, rounds, pb);
        launch_slot_lists(kept_list(c, P, nkept, nullptr), c->p_ub.p, pb, align_round_take(0, rounds), st);
        launches += nkept <= kSlotsSmall ? 2 : 4;
        pb.a_score = c->a_score.p; pb.a_bound = c->a_bound.p; pb.a_tblen = c->a_tblen.p;
        pb.a_pos = c->a_pos.p; pb.a_tb = c->a_tb.p; pb.tbs = tbs;
        // one persistent launch over all kept candidates; scratch for its threads only
        pb.steal = c->tune.align_steal;
        const bool wave = rounds == 1 && nkept <= wave_slots(sp);
        if (!wave && c->scratch.grow(align_workers(nkept, sp) * (int64_t)maxL * wpr)) return STORMGPU_ENOMEM;
        pb.a_scratch = c->scratch.p;
        pb.cells = c->counters.p + kCntAlign;
        if (rounds == 1) {
          if (wave) launch_align_wave(rd, sp, R.d_codes, R.d_mask, 0, nkept, pb, maxL, st);
          else launch_align(rd, sp, R.d_codes, R.d_mask, 0, nkept, pb, st);
          launches++;
        } else {
          // rounds, each of the candidates the replay of the round before selected
          SG_CUDA(cudaEventRecord(c->rev[0], st));
          for (int k = 0; k < rounds; ++k) {
            round_buffers(c, k, pb);
            launch_align(rd, sp, R.d_codes, R.d_mask, 0, nkept, pb, st);
            SG_CUDA(cudaEventRecord(c->rev[2 * k + 1], st));
            launch_replay(n, sp, (int)ref_id, strand ? -1 : 1, pb, align_round_take(k + 1, rounds), out->hits,
                          out->tb, out->tb_stride, out->mapped, st);
            SG_CUDA(cudaEventRecord(c->rev[2 * k + 2], st));
            launches += 2;
          }
        }
        S.aligned += nkept;
      }
      SG_CUDA(cudaEventRecord(c->ev[3], st));
      if (nkept > 0 && rounds == 1) {
        launch_replay(n, sp, (int)ref_id, strand ? -1 : 1, pb, 0, out->hits, out->tb, out->tb_stride, out->mapped, st);
        launches++;
      }
      SG_CUDA(cudaEventRecord(c->ev[4], st));
      SG_CUDA(cudaEventSynchronize(c->ev[4]));
      float a, b, d, e;
      cudaEventElapsedTime(&a, c->ev[0], c->ev[1]);
      cudaEventElapsedTime(&b, c->ev[1], c->ev[2]);
      cudaEventElapsedTime(&d, c->ev[2], c->ev[3]);
      cudaEventElapsedTime(&e, c->ev[3], c->ev[4]);
      if (nkept > 0 && rounds > 1) {  // the rounds' replays count as replay time
        for (int k = 0; k < rounds; ++k) {
          float x = 0;
          cudaEventElapsedTime(&x, c->rev[2 * k + 1], c->rev[2 * k + 2]);
          d -= x;
          e += x;
        }
      }
      tg += a; tf += b; ta += d; tr += e;
      if (nkept > 0) {
        unsigned long long cells = 0;
        SG_CUDA(cudaMemcpyAsync(&cells, c->counters.p + kCntAlign, sizeof(cells), cudaMemcpyDeviceToHost, st));
        SG_CUDA(cudaStreamSynchronize(st));
        S.align_cells += (int64_t)cells;
      }
    }
  }
  SG_CUDA(cudaEventRecord(c->ev[7], st));
  SG_CUDA(cudaEventSynchronize(c->ev[7]));
  SG_CUDA(cudaGetLastError());
  float tt = 0;
  cudaEventElapsedTime(&tt, c->ev[6], c->ev[7]);
  S.ms_gather = tg; S.ms_filter = tf; S.ms_align = ta; S.ms_replay = tr; S.ms_total = tt;
  S.kernels = launches;
  if (n > 0 && wsum > 0) set_densities(c, (double)max_cand / wsum, (double)max_pass / wsum, (double)max_kept / wsum);
  return 0;
}

// Maps reads[lo, hi) into the matching part of out.
static int map_range(stormgpu_ctx* c, const stormgpu_reads* reads, const int16_t* lengths, stormgpu_results* out,
                     int64_t lo, int64_t hi) {
  stormgpu_reads r = *reads;
  stormgpu_results o = *out;
  r.n = hi - lo;
  r.codes += lo * reads->code_stride;
  if (r.levels) r.levels += lo * reads->level_stride;
  r.lengths += lo;
  if (r.first_levels) r.first_levels += lo;
  o.hits += 4 * lo;
  o.tb += 4 * lo * out->tb_stride;
  o.mapped += lo;
  return sg::map_device_impl(c, &r, lengths ? lengths + lo : nullptr, &o);
}

// Maps the batch as consecutive pieces [cuts[q], cuts[q + 1]), the stats summed.
static int map_cuts(stormgpu_ctx* c, const stormgpu_reads* reads, const int16_t* lengths, stormgpu_results* out,
                    const std::vector<int64_t>& cuts) {
  stormgpu_stats acc;
  memset(&acc, 0, sizeof(acc));
  for (size_t q = 0; q + 1 < cuts.size(); ++q) {
    if (cuts[q + 1] <= cuts[q]) continue;
    if (const int e = map_range(c, reads, lengths, out, cuts[q], cuts[q + 1])) return e;
    add_stats(acc, c->stats);
  }
  acc.ms_index = c->stats.ms_index;
  c->stats = acc;
  return 0;
}

// k consecutive pieces of (nearly) equal size
static int map_pieces(stormgpu_ctx* c, const stormgpu_reads* reads, const int16_t* lengths, stormgpu_results* out,
                      int64_t k) {
  std::vector<int64_t> cuts;
  for (int64_t q = 0; q <= k; ++q) cuts.push_back(reads->n * q / k);
  return map_cuts(c, reads, lengths, out, cuts);
}

int sg::map_device_impl(stormgpu_ctx* c, const stormgpu_reads* reads, const int16_t* lengths, stormgpu_results* out) {
  LengthStats ls;
  if (const int e = length_stats(c, reads, lengths, &ls)) return e;
  if (reads->n > 1 && ls.longest <= STORMGPU_MAX_READ_LEN) {
    // at the last call's density per unit of work weight the batch would be cut after its
    // gather: cut it now, into pieces of equal weight (a batch's reads need not be mixed: a file
    // of several lengths often lists them one length after the other).  0.8: the pieces still
    // differ in repeat content; one that overflows is cut after its gather.
    const int64_t n = reads->n;
    const double W = (double)ls.weight;
    const int64_t streams = band_widths(c, make_score_params(c->p)).stream_bytes(n, (int)ls.longest, reads->levels != nullptr);
    const double need = std::max({c->dens_cand * W / (0.8 * (double)kMaxCandidatesPerPass),
                                  c->dens_pass * W / (0.8 * (double)kMaxPassingPerPass),
                                  (double)streams / (double)kMaxStreamBytes});
    if (need > 1.0) {
      std::vector<int16_t> hl;
      if (!lengths) {
        hl.resize(n);
        SG_CUDA(cudaMemcpyAsync(hl.data(), reads->lengths, sizeof(int16_t) * n, cudaMemcpyDeviceToHost, c->st));
        SG_CUDA(cudaStreamSynchronize(c->st));
        lengths = hl.data();
      }
      std::vector<double> cum(n + 1, 0.0);
      for (int64_t r = 0; r < n; ++r) cum[r + 1] = cum[r] + read_weight(lengths[r]);
      const int64_t k = std::min<int64_t>(n, (int64_t)std::ceil(need));
      std::vector<int64_t> cuts(1, 0);
      for (int64_t q = 1; q < k; ++q) {  // strictly increasing, every piece smaller than the batch
        int64_t cut = std::lower_bound(cum.begin(), cum.end(), W * (double)q / (double)k) - cum.begin();
        cut = std::min<int64_t>(std::max<int64_t>(cut, cuts.back() + 1), n - (k - q));
        cuts.push_back(cut);
      }
      cuts.push_back(n);
      return map_cuts(c, reads, lengths, out, cuts);
    }
  }
  int rc;
  const int64_t n = reads->n;
  for (;;) {
    const bool fresh = c->work.used == 0;
    WorkBudget* saved = g_work_budget;
    g_work_budget = &c->work;
    c->work.over = false;
    rc = map_device_once(c, reads, ls, out);
    g_work_budget = saved;
    if (rc != STORMGPU_ENOMEM || !c->work.over) break;
    if (n > 1) {
      rc = kSplitBatch;
      break;
    }
    // A single read with no room beside the buffers that larger batches, given up or of another shape, have
    // left (reads whose streams fill most of the limit): once more without them.
    if (fresh) {
      sg_set_error("one read needs more than the working memory limit of %lld bytes", (long long)c->work.limit);
      return STORMGPU_ENOMEM;
    }
    SG_CUDA(cudaStreamSynchronize(c->st));
    release_work(c);
  }
  if (rc != kSplitBatch) return rc;
  if (n <= 1) {
    sg_set_error("one read has more than %lld candidate diagonals", (long long)kMaxCandidatesPerPass);
    return STORMGPU_ENOMEM;
  }
  return map_pieces(c, reads, lengths, out, 2);
}

extern "C" int stormgpu_map_device(stormgpu_ctx* c, const stormgpu_reads* reads, stormgpu_results* out,
                                   void* stream) {
  if (!c || !reads || !out) { sg_set_error("null argument"); return STORMGPU_EINVAL; }
  SG_CUDA(cudaSetDevice(c->p.device));
  cudaStream_t user = (cudaStream_t)stream;
  if (user) {
    cudaEvent_t e;
    SG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    SG_CUDA(cudaEventRecord(e, user));
    SG_CUDA(cudaStreamWaitEvent(c->st, e, 0));
    cudaEventDestroy(e);
  }
  int rc = map_device_impl(c, reads, nullptr, out);
  if (rc == 0 && user) {
    cudaEvent_t e;
    SG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    SG_CUDA(cudaEventRecord(e, c->st));
    SG_CUDA(cudaStreamWaitEvent(user, e, 0));
    cudaEventDestroy(e);
  }
  return rc;
}

extern "C" int stormgpu_sync(stormgpu_ctx* c) {
  if (!c) return STORMGPU_EINVAL;
  SG_CUDA(cudaStreamSynchronize(c->st));
  return 0;
}

extern "C" int stormgpu_map(stormgpu_ctx* c, const stormgpu_reads* reads, stormgpu_results* out) {
  if (!c || !reads || !out || reads->n < 0) { sg_set_error("null argument"); return STORMGPU_EINVAL; }
  SG_CUDA(cudaSetDevice(c->p.device));
  const int64_t n = reads->n;
  cudaStream_t st = c->st;
  c->last_n = -1;  // the last call's results may go with their buffers: none until this call has its own
  if (c->fcodes.grow(std::max<int64_t>(n * reads->code_stride, 1)) || c->lengths.grow(std::max<int64_t>(n, 1)) ||
      c->hits.grow(std::max<int64_t>(n * 4, 1)) || c->tb.grow(std::max<int64_t>(n * 4 * out->tb_stride, 1)) ||
      c->mapped.grow(std::max<int64_t>(n, 1)))
    return STORMGPU_ENOMEM;
  if (reads->levels && c->flevels.grow(std::max<int64_t>(n * reads->level_stride, 1))) return STORMGPU_ENOMEM;
  if (reads->first_levels && c->first_levels.grow(std::max<int64_t>(n, 1))) return STORMGPU_ENOMEM;
  if (n > 0) {
    SG_CUDA(cudaMemcpyAsync(c->fcodes.p, reads->codes, n * reads->code_stride, cudaMemcpyHostToDevice, st));
    SG_CUDA(cudaMemcpyAsync(c->lengths.p, reads->lengths, sizeof(int16_t) * n, cudaMemcpyHostToDevice, st));
    if (reads->levels) SG_CUDA(cudaMemcpyAsync(c->flevels.p, reads->levels, n * reads->level_stride, cudaMemcpyHostToDevice, st));
    if (reads->first_levels) SG_CUDA(cudaMemcpyAsync(c->first_levels.p, reads->first_levels, n, cudaMemcpyHostToDevice, st));
  }
  stormgpu_reads dr = *reads;
  dr.codes = c->fcodes.p;
  dr.levels = reads->levels ? c->flevels.p : nullptr;
  dr.lengths = c->lengths.p;
  dr.first_levels = reads->first_levels ? c->first_levels.p : nullptr;
  stormgpu_results dres;
  dres.hits = c->hits.p;
  dres.tb = c->tb.p;
  dres.tb_stride = out->tb_stride;
  dres.mapped = c->mapped.p;
  int rc = map_device_impl(c, &dr, reads->lengths, &dres);
  if (rc) return rc;
  c->last_n = n;
  c->last_tbs = out->tb_stride;
  if (n > 0) {
    SG_CUDA(cudaMemcpyAsync(out->hits, c->hits.p, sizeof(stormgpu_hit) * n * 4, cudaMemcpyDeviceToHost, st));
    SG_CUDA(cudaMemcpyAsync(out->tb, c->tb.p, n * 4 * out->tb_stride, cudaMemcpyDeviceToHost, st));
    SG_CUDA(cudaMemcpyAsync(out->mapped, c->mapped.p, n, cudaMemcpyDeviceToHost, st));
  }
  SG_CUDA(cudaStreamSynchronize(st));
  return 0;
}

extern "C" int stormgpu_get_stats(stormgpu_ctx* c, stormgpu_stats* out) {
  if (!c || !out) return STORMGPU_EINVAL;
  *out = c->stats;
  return 0;
}

// ------------------------------------------------------------------------------ unit level

namespace {
int upload_padded(const uint8_t* h, int64_t n_codes, int64_t pad_codes, uint8_t fill, uint8_t** alloc,
                  uint8_t** base) {
  (void)pad_codes;
  const int64_t nb = (n_codes + 3) / 4;
  const int64_t tot = nb + 2 * kPadBytes + 16;
  SG_CUDA(cudaMalloc(alloc, tot));
  SG_CUDA(cudaMemset(*alloc, fill, tot));
  *base = *alloc + kPadBytes;
  if (nb) {
    std::vector<uint8_t> v(h, h + nb);
    for (int64_t k = n_codes; k & 3; ++k) {  // codes past the end: 0 (sequence) or 1 (mask)
      v[k >> 2] &= (uint8_t)~(3u << ((k & 3) << 1));
      if (fill) v[k >> 2] |= (uint8_t)(1u << ((k & 3) << 1));
    }
    SG_CUDA(cudaMemcpy(*base, v.data(), nb, cudaMemcpyHostToDevice));
  }
  return 0;
}
}  // namespace

extern "C" int stormgpu_sw_filter(int W, int read_len, uint32_t match, uint32_t mismatch, uint32_t gapopen,
                                  uint32_t gapext, uint32_t threshold, const uint8_t* genome, int64_t n_codes,
                                  int64_t pad, const int32_t* pos, int64_t n, const uint8_t* read, uint8_t* pass) {
  if (!(W == 2 || W == 4 || W == 8 || W == 16) || read_len <= 0 || read_len > STORMGPU_MAX_READ_LEN || n < 0) {
    sg_set_error("bad filter arguments");
    return STORMGPU_EINVAL;
  }
  for (int64_t k = 0; k < n; ++k)
    if (pos[k] < -(4 * (int64_t)kPadBytes - 64) || pos[k] + read_len + 2 * W > n_codes + 4 * (int64_t)kPadBytes - 64) {
      sg_set_error("window %lld outside the padded genome", (long long)pos[k]);
      return STORMGPU_EINVAL;
    }
  ScoreParams sp;
  memset(&sp, 0, sizeof(sp));
  sp.fm = match & 0xff; sp.fx = mismatch & 0xff; sp.fo = gapopen & 0xff; sp.fe = gapext & 0xff;
  sp.fthr = threshold >= 255u ? 254 : (int)threshold;
  sp.W = W;
  uint8_t *ga, *gb, *dr, *dp;
  int32_t* dpos;
  if (upload_padded(genome, n_codes, pad, 0, &ga, &gb)) return STORMGPU_ECUDA;
  const int rb = (read_len + 2 * W + 16) / 4 + 16;
  std::vector<uint8_t> hr(rb, 0);
  memcpy(hr.data(), read, (read_len + 3) / 4);
  SG_CUDA(cudaMalloc(&dr, rb));
  SG_CUDA(cudaMemcpy(dr, hr.data(), rb, cudaMemcpyHostToDevice));
  SG_CUDA(cudaMalloc(&dpos, sizeof(int32_t) * std::max<int64_t>(n, 1)));
  SG_CUDA(cudaMalloc(&dp, std::max<int64_t>(n, 1)));
  if (n) SG_CUDA(cudaMemcpy(dpos, pos, sizeof(int32_t) * n, cudaMemcpyHostToDevice));
  {
    int16_t L16 = (int16_t)read_len;
    int16_t* dl;
    int32_t* dzero;
    SG_CUDA(cudaMalloc(&dl, sizeof(int16_t)));
    SG_CUDA(cudaMemcpy(dl, &L16, sizeof(int16_t), cudaMemcpyHostToDevice));
    SG_CUDA(cudaMalloc(&dzero, sizeof(int32_t) * std::max<int64_t>(n, 1)));
    SG_CUDA(cudaMemset(dzero, 0, sizeof(int32_t) * std::max<int64_t>(n, 1)));
    uint8_t *gx, *rx;
    const int64_t rstride = rexp_stride(read_len);
    SG_CUDA(cudaMalloc(&gx, n_codes + 2 * kGexpPad + 16));
    SG_CUDA(cudaMemset(gx, 0, n_codes + 2 * kGexpPad + 16));
    SG_CUDA(cudaMalloc(&rx, rstride));
    launch_expand_genome(gb, n_codes, gx + kGexpPad, 0);
    ReadsDev one{1, dr, rb, nullptr, 0, dl};
    launch_expand_reads(one, rx, rstride, 0);
    FilterJob job;
    memset(&job, 0, sizeof(job));
    job.n = n; job.fr = dzero; job.fd = dpos; job.flag = dp; job.codes = dr; job.cstride = rb;
    job.lengths = dl; job.genome = gb; job.W = W; job.Is = 0;
    job.gexp = gx + kGexpPad; job.rexp = rx; job.rstride = rstride; job.min_len = read_len;
    job.fm = sp.fm; job.fx = sp.fx; job.fo = sp.fo; job.fe = sp.fe; job.fthr = sp.fthr;
    job.band = band_filter_consts(sp.fm, sp.fx, sp.fo, sp.fe, sp.fthr);
    job.band_H = filter_band_registers(W, job.band);
    uint32_t* bs = nullptr;
    if (job.band_H) {
      job.bwords = band_stream_words(read_len, job.band_H);
      SG_CUDA(cudaMalloc(&bs, job.bwords * sizeof(uint32_t)));
      launch_band_streams(one, job.band_H, job.bwords, bs, nullptr, job.band, 0);
      job.bs = bs;
    }
    launch_filter_flat_job(job, sp, filter_dpx_ok(sp, read_len), 0);
    SG_CUDA(cudaGetLastError());
    SG_CUDA(cudaDeviceSynchronize());
    cudaFree(dl);
    cudaFree(dzero);
    cudaFree(gx);
    cudaFree(rx);
    if (bs) cudaFree(bs);
  }
  SG_CUDA(cudaGetLastError());
  SG_CUDA(cudaDeviceSynchronize());
  if (n) SG_CUDA(cudaMemcpy(pass, dp, n, cudaMemcpyDeviceToHost));
  cudaFree(ga); cudaFree(dr); cudaFree(dpos); cudaFree(dp);
  return 0;
}

extern "C" int stormgpu_align(const stormgpu_params* params, const uint8_t* read, const uint8_t* levels,
                              int read_len, const uint8_t* genome, const uint8_t* mask, int64_t n_codes,
                              int64_t pad, const int32_t* win, int64_t n, int32_t* score, int32_t* bound,
                              int16_t* best, int32_t* tb_len, uint8_t* tb, int64_t tb_stride) {
  if (!params || read_len <= 0 || read_len > STORMGPU_MAX_READ_LEN || n < 0 ||
      params->allowed_indels < 0 || params->allowed_indels > STORMGPU_MAX_INDELS) {
    sg_set_error("bad align arguments");
    return STORMGPU_EINVAL;
  }
  const int I = params->allowed_indels;
  if (tb_stride < (read_len + I + 1) / 2) { sg_set_error("tb_stride too small"); return STORMGPU_EINVAL; }
  for (int64_t k = 0; k < n; ++k)
    if (win[k] < -(4 * (int64_t)kPadBytes - 64) || win[k] + read_len + 2 * I > n_codes + 4 * (int64_t)kPadBytes - 64) {
      sg_set_error("window outside the padded genome");
      return STORMGPU_EINVAL;
    }
  ScoreParams sp = make_score_params(*params);
  sp.Is = 1 << 28;              // window = diag - I exactly
  sp.min_score = -(1 << 29);    // always trace back
  sp.packed = sp.small ? 2 : 0;  // every cell exact: the packed form where no cell meets its floor
  uint8_t *ga, *gb, *ma, *mb;
  if (upload_padded(genome, n_codes, pad, 0, &ga, &gb)) return STORMGPU_ECUDA;
  if (upload_padded(mask, n_codes, pad, 0x55, &ma, &mb)) return STORMGPU_ECUDA;
  const int64_t rb = ((read_len + 3) / 4 + 15) & ~7;
  std::vector<uint8_t> hr(rb, 0), hq(rb, 0);
  memcpy(hr.data(), read, (read_len + 3) / 4);
  if (levels) memcpy(hq.data(), levels, (read_len + 3) / 4);
  uint8_t *dr, *dq = nullptr;
  int16_t* dl;
  SG_CUDA(cudaMalloc(&dr, rb));
  SG_CUDA(cudaMemcpy(dr, hr.data(), rb, cudaMemcpyHostToDevice));
  if (levels) {
    SG_CUDA(cudaMalloc(&dq, rb));
    SG_CUDA(cudaMemcpy(dq, hq.data(), rb, cudaMemcpyHostToDevice));
  }
  int16_t L16 = (int16_t)read_len;
  SG_CUDA(cudaMalloc(&dl, sizeof(int16_t)));
  SG_CUDA(cudaMemcpy(dl, &L16, sizeof(int16_t), cudaMemcpyHostToDevice));
  ReadsDev rd{1, dr, rb, dq, rb, dl};
  PassBuffers pb;
  memset(&pb, 0, sizeof(pb));
  const int64_t nn = std::max<int64_t>(n, 1);
  const int BW = 2 * I + 1;
  const int wpr = (2 * BW + 31) / 32 + (params->colour ? (BW + 31) / 32 : 0);
  const int64_t tbs = ((read_len + I + 1) / 2 + 7) & ~7LL;
  std::vector<int32_t> zeros(nn, 0), diag(nn, 0);
  for (int64_t k = 0; k < n; ++k) diag[k] = win[k] + I;
  SG_CUDA(cudaMalloc(&pb.p_read, sizeof(int32_t) * nn));
  SG_CUDA(cudaMalloc(&pb.p_diag, sizeof(int32_t) * nn));
  SG_CUDA(cudaMalloc(&pb.a_score, sizeof(int32_t) * nn));
  SG_CUDA(cudaMalloc(&pb.a_bound, sizeof(int32_t) * nn));
  SG_CUDA(cudaMalloc(&pb.a_tblen, sizeof(int32_t) * nn));
  SG_CUDA(cudaMalloc(&pb.a_pos, sizeof(int16_t) * 4 * nn));
  SG_CUDA(cudaMalloc(&pb.a_tb, tbs * nn));
  SG_CUDA(cudaMalloc(&pb.a_scratch, sizeof(uint32_t) * (size_t)read_len * wpr * nn));
  pb.tbs = tbs;
  SG_CUDA(cudaMemcpy(pb.p_read, zeros.data(), sizeof(int32_t) * nn, cudaMemcpyHostToDevice));
  SG_CUDA(cudaMemcpy(pb.p_diag, diag.data(), sizeof(int32_t) * nn, cudaMemcpyHostToDevice));
  if (n <= wave_slots(sp)) launch_align_wave(rd, sp, gb, mb, 0, n, pb, read_len, 0);
  else launch_align(rd, sp, gb, mb, 0, n, pb, 0);
  SG_CUDA(cudaGetLastError());
  SG_CUDA(cudaDeviceSynchronize());
  if (n) {
    SG_CUDA(cudaMemcpy(score, pb.a_score, sizeof(int32_t) * n, cudaMemcpyDeviceToHost));
    SG_CUDA(cudaMemcpy(bound, pb.a_bound, sizeof(int32_t) * n, cudaMemcpyDeviceToHost));
    SG_CUDA(cudaMemcpy(best, pb.a_pos, sizeof(int16_t) * 4 * n, cudaMemcpyDeviceToHost));
    SG_CUDA(cudaMemcpy(tb_len, pb.a_tblen, sizeof(int32_t) * n, cudaMemcpyDeviceToHost));
    std::vector<uint8_t> htb(tbs * n);
    SG_CUDA(cudaMemcpy(htb.data(), pb.a_tb, tbs * n, cudaMemcpyDeviceToHost));
    for (int64_t k = 0; k < n; ++k) {
      memset(tb + k * tb_stride, 0, tb_stride);
      memcpy(tb + k * tb_stride, htb.data() + k * tbs, std::min<int64_t>(tbs, tb_stride));
    }
  }
  cudaFree(ga); cudaFree(ma); cudaFree(dr); if (dq) cudaFree(dq); cudaFree(dl);
  cudaFree(pb.p_read); cudaFree(pb.p_diag); cudaFree(pb.a_score); cudaFree(pb.a_bound);
  cudaFree(pb.a_tblen); cudaFree(pb.a_pos); cudaFree(pb.a_tb); cudaFree(pb.a_scratch);
  return 0;
}

extern "C" int stormgpu_index_one(const char* seed, int32_t stdev_distance, const uint8_t* codes, int64_t n_codes,
                                  int64_t pad, const int32_t* rs, const int32_t* re, int32_t n_regions,
                                  int32_t* first, int32_t* map, int64_t map_capacity, int64_t* map_len) {
  SeedSet ss;
  if (parse_seeds(seed, &ss) != 0 || ss.n < 1) { sg_set_error("invalid seed"); return STORMGPU_EINVAL; }
  uint8_t *ga, *gb;
  if (upload_padded(codes, n_codes, pad, 0, &ga, &gb)) return STORMGPU_ECUDA;
  DevIndex ix;
  int rc = build_indexes(gb, n_codes, rs, re, n_regions, ss.s, 1, stdev_distance, &ix, 0, nullptr);
  if (rc) { cudaFree(ga); return rc; }
  SG_CUDA(cudaDeviceSynchronize());
  SG_CUDA(cudaMemcpy(first, ix.first, sizeof(int32_t) * (ix.nkeys + 1), cudaMemcpyDeviceToHost));
  if (ix.n > map_capacity) { sg_set_error("map_capacity too small"); cudaFree(ga); return STORMGPU_EINVAL; }
  if (ix.n) SG_CUDA(cudaMemcpy(map, ix.map, sizeof(int32_t) * ix.n, cudaMemcpyDeviceToHost));
  *map_len = ix.n;
  cudaFree(ix.first);
  if (ix.map) cudaFree(ix.map);
  cudaFree(ga);
  return 0;
}
