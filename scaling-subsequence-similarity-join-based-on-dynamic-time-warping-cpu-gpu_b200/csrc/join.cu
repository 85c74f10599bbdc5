// Host orchestration of the join and the C ABI (include/dtwj.h).
//
// The reference's driver (GPU_version1/src/new_dtw_motifGUI_malloc.cu:30-816)
// prepares everything on the host, allocates one device buffer per
// subsequence and then loops over diagonal blocks with five launches and
// three host synchronisations per block.  Here every phase runs on one
// stream with device-resident state:
//   prep      statistics, envelopes, mask, row constants        (prep.cu)
//   profile   ED matrix profile, row minima                      (mp.cu)
//   seeds     kSeeds smallest profile entries -> exact DTW        (mp.cu, pairs.cu)
//   sweep     per chunk of tiles: group bound, diagonal bound on the tiles it
//             leaves dense -> block-mean / endpoint / LB_Keogh /
//             DTW                          (group.cu, lb.cu, paa.cu, runs.cu, pairs.cu)
//   verify    FP64 DTW of every candidate near the final best     (pairs.cu)
// with a single host synchronisation at the end.
#include "../../include/dtwj.h"
#include "dtwj_dev.cuh"

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

using namespace dtwj;

namespace {

constexpr unsigned int kCandCap = 1u << 20;
constexpr unsigned int kQueueCapMax = 1u << 26;
// Default tiles per chunk of the sweep: kLbChunkRounds tiles for each of the
// diagonal sweep's resident CTAs, chosen when that bound ran on every tile (1M
// bench series: 0.973 s per join at 4 rounds, 0.998 at 3, 0.980 at 5).  Tiles
// that the group bound leaves sparse skip it, and each stage's tail is then what
// a chunk costs: 157 ms at 444 tiles, 136 at 888, 119 at 1332, 112 at 1776, 103
// at 2664, 97 at 4096 (dtwj_ctx_set_tuning).  The survivor bits, 451 KB for every
// tile of a chunk, are what larger chunks cost.
constexpr int kLbChunkRounds = 4;
// Largest piece an overflowing chunk is swept again in.  Every piece that
// overflows again wastes a full DTW queue of work.  On the 262,144-sample
// ECG-like series at w = 103 nearly every pair reaches LB_Keogh, about 3.5
// million per tile by that join's stage counts, so 32 tiles fit the LB_Keogh
// queue (2^27 entries) and 55 would not.
constexpr int kResweepTiles = 32;
// Tiles from which the seeds come from the group bound instead of a walk over
// every diagonal: random walks of 100,003 samples (1,421 tiles, m = 256) 0.87 ms
// against 1.04, of 131,071 (m = 512) 1.02 against 1.74; at 65,536 (590 tiles)
// 0.62 against 0.56.
constexpr int kSeedGroupTiles = 1024;
// Tiles from which a sample decides whether the sweep uses the group bound at all:
// 3 us, where a join of a random walk takes 0.7 ms and more; noise of 30,000
// samples (144 tiles, m = 64, w = 0) takes 1.3 ms with it and 3.8 without.
constexpr int kProbeTiles = 128;
// Their lists of group pairs, and with the samples and five words the bytes
// they take.
constexpr unsigned int kSeedSupCap = 1u << 24, kSeedListCap = 1u << 22;
constexpr size_t kSeedScratch =
    (size_t)kSeedSupCap * 4 + (size_t)kSeedListCap * sizeof(uint2) + kSeedSamples * 4 + 64;
// Largest window table (three FP32 rows per window).
constexpr size_t kWindowTableMax = (size_t)2 << 30;
// (m, w) groups of a batch joined at the same time, one context each.
constexpr int kBatchWorkers = 4;

// Status bits: 1 input not finite, 2 a queue overflowed in the current chunk,
// 8 one did in an earlier chunk of this sweep.
constexpr int kOverflowSeen = 8;

struct Buf {
  void* p = nullptr;
  size_t cap = 0;
};

struct Timer {
  std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
  double seconds() const {
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  }
};

// What one chunk of the sweep left behind: whether one of its queues
// overflowed (pairs were dropped, so the chunk is swept again), and the
// counters after it, so that a chunk swept again can be taken out of them.
struct ChunkNote {
  unsigned long long counters[kNumCounters];
  unsigned int overflow;
  unsigned int pad;
};

// Sort keys of the learned order: ascending score, NaN last; the radix sort
// is stable, so ties keep the plain order.
__global__ void k_order_keys(const float* score, int n, unsigned int* key, int* idx) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float f = score[t];
  const unsigned int u = __float_as_uint(f);
  key[t] = f != f ? 0xffffffffu : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
  idx[t] = t;
}

// Tiles in the sorted order, each with its position.
__global__ void k_gather_tiles(const Tile* plain, const int* idx, int n, Tile* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  Tile x = plain[idx[t]];
  x.order = t;
  out[t] = x;
}

// Runs after a chunk's last stage on the join's stream: notes the chunk and
// clears the overflow bit for the next one.
__global__ void k_chunk_note(int* status, const unsigned long long* counters, ChunkNote* note) {
  const int t = threadIdx.x;
  if (t < kNumCounters) note->counters[t] = counters[t];
  if (t == 0) {
    const int s = *status;
    note->overflow = (s & 2) ? 1u : 0u;
    *status = (s & 2) ? (s & ~2) | kOverflowSeen : s;
  }
}

// The search state of a join before its first DTW: best-so-far +inf per slot,
// counters, candidates and the seeds' work counter zero.
__global__ void k_init_search(unsigned int* bsf2, int nslots, unsigned long long* counters,
                              unsigned int* cand_count, unsigned int* nseeds, int nseries,
                              int seed_slots, unsigned int* zready, unsigned int* low,
                              unsigned int* probe) {
  for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < nslots; x += gridDim.x * blockDim.x)
    bsf2[x] = 0x7f800000u;
  if (blockIdx.x == 0) {
    if (threadIdx.x < kNumCounters) counters[threadIdx.x] = 0ull;
    if (threadIdx.x == 0) {
      *cand_count = 0u;
      nseeds[nseries] = (unsigned int)seed_slots;
      nseeds[nseries + 1] = 0u;
      zready[0] = zready[1] = 0u;  // the window table: not filled
      low[0] = 64u;  // at least 129 are pruned before all are tried
      low[1] = 0u;
      probe[0] = probe[1] = 0u;
    }
  }
}

}  // namespace

struct dtwj_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 0;
  std::vector<Buf> bufs;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::vector<Tile> lbtiles_host;    // kLbLags-lag tiles of the diagonal sweep
  int64_t lbtiles_n = -1, lbtiles_m = -1;  // single-series shape the tiles were built for
  // what the plain tiles on the device are those of (a single series' join)
  struct TilesKey {
    const void* p;
    int64_t n, m;
    int rank, world;
  } tiles_dev = {nullptr, -1, -1, 0, 1};
  // staging of a call's results.  Pageable: pinning 64 KB once per context took
  // 5 ms and gained 8 us a join (2,000 samples: 350 -> 341 us)
  std::vector<unsigned char> staging;
  std::vector<Tile> tiles_run;             // the tiles in the order of the current call
  dtwj_mlp* model = nullptr;               // scores tiles for DTWJ_F_LEARNED (not owned)
  std::vector<std::pair<int, BandShape>> band_override;  // band w -> DTW layout (autotuner)
  int dtw_warps = 0;    // CTA size of the join's DTW kernel in warps (0: default)
  int chunk_tiles = 0;  // tiles per chunk of the sweep (0: default)
  int shard_rank = 0, shard_world = 1;  // this context sweeps tiles t with t % world == rank
  dtwj_exchange_fn exchange = nullptr;  // best-so-far exchange between sweep phases
  void* exchange_user = nullptr;
  int exchange_phases = 0;
  std::vector<cudaEvent_t> pool;  // events for per-phase device times
  // the sweep's launches captured as a CUDA graph, replayed while every
  // launch argument is unchanged (same buffers, tiles, band, flags)
  cudaGraphExec_t sweep_exec = nullptr;
  std::vector<unsigned char> sweep_key;
  std::vector<unsigned char> sweep_seen;  // the last launches made directly
  std::vector<int> sweep_marks;  // phase marks of the capture: (phase, a, b, launches)
  size_t sweep_ev0 = 0, sweep_ev1 = 0;
};

namespace {

enum BufId {
  B_A = 0, B_WORK, B_RESULT, B_PAIRS, B_OUT, B_LBTILES, B_TILEBEST, B_FEAT, B_SCORE, B_NOTES2,
  B_SORT, B_SORT_TEMP, B_LBTILES2,
  B_COUNT_
};

int ensure(dtwj_ctx* c, int id, size_t bytes, void** out) {
  if (c->bufs.size() < (size_t)B_COUNT_) c->bufs.resize(B_COUNT_);
  Buf& b = c->bufs[id];
  if (b.cap < bytes) {
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.cap = 0;
    size_t want = bytes < 256 ? 256 : bytes;
    if (cudaMalloc(&b.p, want) != cudaSuccess) {
      cudaGetLastError();
      return DTWJ_ERR_OOM;
    }
    b.cap = want;
  }
  *out = b.p;
  return DTWJ_OK;
}

#define ENSURE(id, bytes, ptr)                                       \
  do {                                                               \
    void* _p = nullptr;                                              \
    int _rc = ensure(ctx, id, (size_t)(bytes), &_p);                 \
    if (_rc) return _rc;                                             \
    ptr = reinterpret_cast<decltype(ptr)>(_p);                       \
  } while (0)

// Several arrays in one device buffer, each on a 256-byte boundary.  An
// allocation and its release cost 0.7 ms at 10 MB and 2.3 ms at 2 GB, which a
// one-shot call pays every time: with one buffer, and queues no longer than
// the series has pairs, the one-shot ECG-like join of 9,001 samples takes 12.8
// ms (10.6 of them on the device), with a buffer per array it took 17, and 22
// with pinned staging made for a single call.
struct Arena {
  std::vector<std::pair<void**, size_t>> parts;
  template <typename T>
  void add(T** p, size_t bytes) {
    parts.push_back({reinterpret_cast<void**>(p), bytes});
  }
  int place(dtwj_ctx* ctx, int id) {
    size_t total = 0;
    for (auto& q : parts) total += (q.second + 255) / 256 * 256;
    void* base = nullptr;
    const int rc = ensure(ctx, id, total, &base);
    if (rc) return rc;
    unsigned char* at = static_cast<unsigned char*>(base);
    for (auto& q : parts) {
      *q.first = at;
      at += (q.second + 255) / 256 * 256;
    }
    return DTWJ_OK;
  }
};

#define CUDA_OK(expr)                                                 \
  do {                                                                \
    cudaError_t _e = (expr);                                          \
    if (_e != cudaSuccess) {                                          \
      if (getenv("DTWJ_DEBUG"))                                       \
        fprintf(stderr, "dtwj: %s failed: %s\n", #expr, cudaGetErrorString(_e)); \
      return DTWJ_ERR_CUDA;                                           \
    }                                                                 \
  } while (0)

// Per-phase device time from CUDA events recorded on the join's stream
// (DTWJ_F_PROFILE); a no-op otherwise.
struct Phases {
  dtwj_ctx* ctx;
  bool on;
  size_t used = 0;
  struct Mark {
    int phase;
    size_t a, b;
    int launches;
  };
  std::vector<Mark> marks;
  size_t open_at = 0;
  Phases(dtwj_ctx* c, bool enabled) : ctx(c), on(enabled) {}
  cudaEvent_t ev(size_t k) {
    while (ctx->pool.size() <= k) {
      cudaEvent_t e;
      cudaEventCreate(&e);
      ctx->pool.push_back(e);
    }
    return ctx->pool[k];
  }
  // While the stream is being captured, records are external: they become
  // event-record nodes of the graph (a plain record would only order the
  // capture, and the external flag is refused outside a capture).
  bool capturing = false;
  void record(cudaEvent_t e) {
    if (capturing) cudaEventRecordWithFlags(e, ctx->stream, cudaEventRecordExternal);
    else cudaEventRecord(e, ctx->stream);
  }
  void begin() {
    if (!on) return;
    open_at = used;
    record(ev(used++));
  }
  void end(int phase, int launches) {
    if (!on) return;
    record(ev(used));
    marks.push_back({phase, open_at, used, launches});
    ++used;
  }
  void collect(dtwj_result* out) {
    for (auto& mk : marks) {
      float ms = 0.f;
      if (cudaEventElapsedTime(&ms, ctx->pool[mk.a], ctx->pool[mk.b]) != cudaSuccess) {
        cudaGetLastError();  // a mark without a time must not fail the next call
        ms = 0.f;
      }
      out->phase_seconds[mk.phase] += ms / 1000.0;
      out->phase_launches[mk.phase] += (uint64_t)mk.launches;
    }
  }
};

int check_args(const void* x, int64_t n, int32_t m, int32_t w) {
  if (!x || m < 8 || m > DTWJ_MAX_M || w < 0) return DTWJ_ERR_ARG;
  if (n < 2 * (int64_t)m + 1 || n > (int64_t)INT32_MAX - 4) return DTWJ_ERR_ARG;
  return DTWJ_OK;
}

// Tiles of the profile and the diagonal sweep (kLbLags lags x kLbRows rows)
// for every series; a single series keeps its tiles across calls.
void build_lb_tiles(dtwj_ctx* ctx, int64_t n, int m, const int64_t* sbeg, int nseries) {
  if (!sbeg && ctx->lbtiles_n == n && ctx->lbtiles_m == m) return;
  ctx->lbtiles_host.clear();
  int32_t order = 0;
  for (int r = 0; r < nseries; ++r) {
    const int64_t wb = sbeg ? sbeg[r] : 0;
    const int64_t s = (sbeg ? sbeg[r + 1] - sbeg[r] : n) - m + 1;
    for (int64_t L0 = m; L0 <= s - 1; L0 += kLbLags) {
      const int64_t rows_total = s - L0;
      for (int64_t i0 = 0; i0 < rows_total; i0 += kLbRows) {
        Tile t;
        t.L0 = (int32_t)L0;
        t.i0 = (int32_t)(wb + i0);
        t.rows = (int32_t)(rows_total - i0 < kLbRows ? rows_total - i0 : kLbRows);
        t.order = order++;
        t.send = (int32_t)(wb + s);
        t.series = r;
        ctx->lbtiles_host.push_back(t);
      }
    }
  }
  ctx->lbtiles_n = sbeg ? -1 : n;
  ctx->lbtiles_m = sbeg ? -1 : m;
}

// Host memory for a copy of `bytes` from the device, valid until the next one.
unsigned char* staging(dtwj_ctx* ctx, size_t bytes) {
  if (ctx->staging.size() < bytes) ctx->staging.resize(bytes);
  return ctx->staging.data();
}

// How much of a series prepare() makes: the window statistics (pair lists),
// also the update terms of the covariance recurrence (the matrix profile),
// also the envelopes and everything a sweep reads, also the records of the
// group filter (joins).
enum Prep { kPrepStats, kPrepProfile, kPrepSweep, kPrepJoin };

// What the preparation needs besides the DevSeries' own arrays.
struct PrepScratch {
  bool masked = false;
  Prep level = kPrepStats;
  const int64_t* sbeg_host = nullptr;
  int64_t* sbeg = nullptr;
  int* sid = nullptr;
  double* gmeans = nullptr;
  unsigned int* counts = nullptr;
  double *diff = nullptr, *mean = nullptr;
  float* zmax = nullptr;
};

// Lays out the per-series arrays in A (not placed yet).  A batch (sbeg !=
// nullptr) holds nseries series back to back in x_dev, series r on samples
// [sbeg[r], sbeg[r + 1]).  The group filter's records are made where the
// single-pair block-mean bound reads one offset per window (m <= 1024);
// without them every tile goes through the diagonal bound.
void plan_series(Arena& A, const double* x_dev, int64_t n, int m, int w, bool masked, Prep level,
                 const int64_t* sbeg_host, int nseries, DevSeries* S, PrepScratch* P) {
  const int64_t s = n - m + 1;
  memset(S, 0, sizeof *S);
  S->a = x_dev;
  S->n = n;
  S->s = s;
  S->m = m;
  S->w = w;
  S->nseries = nseries;
  P->masked = masked;
  P->level = level;
  P->sbeg_host = sbeg_host;
  if (sbeg_host) {
    A.add(&P->sbeg, (size_t)(nseries + 1) * 8);
    A.add(&P->sid, (size_t)n * 4);
  }
  A.add(&S->mu, s * 8);
  A.add(&S->sig, s * 8);
  A.add(&S->isg, s * 8);
  A.add(&S->flat, s);
  if (level >= kPrepProfile) {
    A.add(&S->dfa, s * 8);
    A.add(&S->dga, s * 8);
  }
  if (level >= kPrepSweep) {
    A.add(&S->U, n * 8);
    A.add(&S->L, n * 8);
    A.add(&S->E, n * 8);
    A.add(&S->nu, s * 8);
    A.add(&S->dfE, s * 8);
    A.add(&S->dgE, s * 8);
    A.add(&S->A, s * 8);
    A.add(&S->DUL, s * 8);
    A.add(&S->qsig, s * 8);
    A.add(&S->cb, ((n >> kBlkShift) + 4) * 8);
    A.add(&S->af, n * 4);
    A.add(&S->ulf, n * 8);
    S->paa_b = paa_block(m);
    if (m <= (1 << kBlkShift)) {
      A.add(&S->pq2, (size_t)n * 32);
      const int fine = S->paa_b / 4;
      S->fine_n = n / fine + 2;
      A.add(&S->fq, (size_t)S->fine_n * fine * 2 * sizeof(float));
      A.add(&S->ful, (size_t)S->fine_n * fine * 2 * sizeof(float2));
      A.add(&S->cmax2, (size_t)kCopyBlocks(n) * 8);
      A.add(&S->wrec, (size_t)s * 16);
    } else {
      A.add(&S->pq, (size_t)n * 16);
    }
    A.add(&S->cmax, ((n >> kBlkShift) + 4) * 4);
    A.add(&S->rw, s * 4);
  }
  if (masked) {
    A.add(&S->mask, n * 4);
    A.add(&S->MN, s * 4);
    A.add(&S->MDUL2, s * 4);
    A.add(&S->MDUL, s * 4);
    A.add(&S->SM, s * 8);
    A.add(&S->SME, s * 8);
    A.add(&P->zmax, 4);
    A.add(&P->counts, (size_t)m * mask_table_max(m) * 4);
    A.add(&P->diff, n * 8);
    A.add(&P->mean, 8);
  }
  if (level >= kPrepJoin && m <= (1 << kBlkShift)) {
    group_shape(m, s, S);
    A.add(&S->grp, (size_t)S->grp_n * S->grp_d * sizeof(float4));
    A.add(&S->sup, (size_t)S->sup_n * S->grp_d * sizeof(float4));
    A.add(&P->gmeans, (size_t)n * 24);
  }
  A.add(&S->status, 4);
}

// Prepares the planned and placed arrays.
int prepare(dtwj_ctx* ctx, DevSeries& S, const PrepScratch& P, Phases* ph = nullptr) {
  const int m = S.m;
  const bool masked = P.masked;
  const Prep level = P.level;
  const int64_t* sbeg_host = P.sbeg_host;
  if (sbeg_host) {
    CUDA_OK(cudaMemcpyAsync(P.sbeg, sbeg_host, (size_t)(S.nseries + 1) * 8, cudaMemcpyHostToDevice,
                            ctx->stream));
    launch_series_ids(P.sbeg, S.nseries, P.sid, S.n, ctx->stream);
    S.sbeg = P.sbeg;
    S.sid = P.sid;
  }
  cudaStream_t st = ctx->stream;
  // the input's check, waited for before anything reads the series
  int verdict = 0;
  CUDA_OK(cudaMemsetAsync(S.status, 0, 4, st));
  launch_check_finite(S.a, S.n, S.status, st);
  CUDA_OK(cudaMemcpyAsync(&verdict, S.status, 4, cudaMemcpyDeviceToHost, st));
  CUDA_OK(cudaStreamSynchronize(st));
  if (verdict & 1) return DTWJ_ERR_NAN;
  if (ph) ph->begin();
  int launches = 1;
  if (level < kPrepSweep) {
    launch_stats(S, st);
    if (level == kPrepProfile) launches += launch_diffs(S, st);
  } else {
    launch_prep(S, st);
    if (masked) {
      const int lt_max = mask_table_max(m);
      unsigned int* counts = P.counts;
      double *diff = P.diff, *mean = P.mean;
      float* zmax = P.zmax;
      if (!sbeg_host) {
        launch_mask(S, counts, lt_max, diff, mean, zmax, st);
      } else {
        // the mask's CDF tables are per series: build it on a view of each one
        for (int r = 0; r < S.nseries; ++r) {
          const int64_t b = sbeg_host[r], nr = sbeg_host[r + 1] - b;
          DevSeries V = S;
          V.a = S.a + b;
          V.n = nr;
          V.s = nr - m + 1;
          V.mu = S.mu + b;
          V.sig = S.sig + b;
          V.isg = S.isg + b;
          V.flat = S.flat + b;
          V.U = S.U + b;
          V.L = S.L + b;
          V.mask = S.mask + b;
          V.sid = nullptr;
          V.sbeg = nullptr;
          V.nseries = 1;
          launch_mask(V, counts, lt_max, diff, mean, zmax, st);
        }
      }
    }
    launch_rowterms(S, masked, st);
    launch_center(S, st);
    launches = (masked ? 11 : 6) + launch_paa_prep(S, st);
    if (S.grp) launches += launch_group_prep(S, P.gmeans, st);
  }
  if (ph) ph->end(DTWJ_PHASE_PREP, launches);
  CUDA_OK(cudaGetLastError());
  return DTWJ_OK;
}

// The same in one, for calls that need no other buffers of the arena.
int plan_and_prepare(dtwj_ctx* ctx, const double* x_dev, int64_t n, int m, int w, bool masked,
                     Prep level, DevSeries* S, PrepScratch* P) {
  Arena A;
  plan_series(A, x_dev, n, m, w, masked, level, nullptr, 1, S, P);
  const int rc = A.place(ctx, B_WORK);
  return rc ? rc : prepare(ctx, *S, *P);
}

int effective_band(int m, int w) { return w > m - 1 ? m - 1 : w; }

// Per-tile outputs of dtwj_ctx_tiles (host arrays, one entry per tile).
struct TileQuery {
  float* features;   // [tiles][64] or nullptr
  double* min_dist;  // exact smallest DTW distance per tile, or nullptr
};

// Joins one series (sbeg == nullptr, nseries == 1) or a batch of nseries
// series of one (m, w) stored back to back (series r on samples
// [sbeg[r], sbeg[r + 1])); outs[r] receives series r's top-1 pair with
// indices relative to its own first sample.  With tq (one series) the call
// reports per-tile values instead of a join: the tile features, and with
// tq->min_dist the exact smallest DTW distance of every tile, found by a sweep
// in which every tile prunes against its own best-so-far only.
int run_join(dtwj_ctx* ctx, const double* x_dev, int64_t n, const int64_t* sbeg, int nseries,
             int32_t m, int32_t w_in, uint32_t flags, dtwj_result* outs, double t_upload,
             const TileQuery* tq = nullptr) {
  Timer wall;
  const int w = effective_band(m, w_in);
  BandShape band;
  if (!choose_band_join(m, w, &band)) return DTWJ_ERR_BAND;
  for (const auto& bo : ctx->band_override)
    if (bo.first == w) band = bo.second;
  band.warps = ctx->dtw_warps;
  // the seeds and the verification: few pairs, each as fast as one can go
  BandShape wide;
  choose_band(w, &wide);
  // windows too long for the FP64 verification (features need none)
  if (!(tq && !tq->min_dist) && !pair_list_fits(m, wide, true)) return DTWJ_ERR_ARG;
  const bool learned = (flags & DTWJ_F_LEARNED) && !tq;
  if (learned && !ctx->model) return DTWJ_ERR_NOMODEL;
  if (learned && mlp_device(ctx->model) != ctx->device) return DTWJ_ERR_ARG;
  const bool tile_mode = tq && tq->min_dist;
  // the run filter: the block-mean bound (default), or the reference's masked
  // diagonal bound and endpoint bound (DTWJ_F_MASKED_CASCADE)
  const bool cascade = (flags & DTWJ_F_MASKED_CASCADE) != 0;
  const bool masked = cascade && !(flags & DTWJ_F_NO_MASKED) && !(flags & DTWJ_F_NO_DIAG);
  const bool verbose = flags & DTWJ_F_VERBOSE;
  // LB_Petitjean between LB_Keogh and DTW, where its shared tables fit
  const bool petitjean = (flags & DTWJ_F_PETITJEAN) && !(flags & DTWJ_F_NO_DIAG) &&
                         petitjean_fits(m, w);
  cudaStream_t st = ctx->stream;
  Phases ph(ctx, (flags & DTWJ_F_PROFILE) != 0);
  CUDA_OK(cudaEventRecord(ctx->ev0, st));

  // tiles of the sweep; a single series' stay on the device while its shape and
  // shard do
  const int world = tq ? 1 : ctx->shard_world, rank = tq ? 0 : ctx->shard_rank;
  std::vector<Tile>& th = ctx->tiles_run;
  const auto& tk = ctx->tiles_dev;
  const bool keep_tiles = !sbeg && !tile_mode && tk.p && tk.p == ctx->bufs[B_LBTILES].p &&
                          tk.n == n && tk.m == m && tk.rank == rank && tk.world == world;
  if (!keep_tiles) {
    ctx->tiles_dev.p = nullptr;  // until the new ones are on their way
    build_lb_tiles(ctx, n, m, sbeg, nseries);
    th = ctx->lbtiles_host;
    if (world > 1) {
      // one shard of the tiles (round robin): the profile, the seeds and the
      // sweep only see these; the shards' results combine by their minimum
      size_t k = 0;
      for (size_t t = 0; t < th.size(); ++t)
        if ((int)(t % (size_t)world) == rank) th[k++] = th[t];
      th.resize(k);
    }
  }
  const int nlb = (int)th.size();
  // best-so-far slots: one per series, or one per tile for the tile minima
  const int nslots = tile_mode ? (nlb > 0 ? nlb : 1) : nseries;

  // what the call returns, in one block: [nslots] best_d2, best_ij, best_f32,
  // seed_bsf, then the counters, the candidate count and the status word
  unsigned long long *best_d2, *best_ij;
  float* best_f32;
  unsigned int* seed_bsf;
  DevSearch Q;
  memset(&Q, 0, sizeof Q);
  int* status_dev;
  const size_t at_counters = ((size_t)nslots * 24 + 7) / 8 * 8;
  const size_t result_bytes = at_counters + kNumCounters * 8 + 8;
  unsigned char* result_dev;
  ENSURE(B_RESULT, result_bytes, result_dev);
  best_d2 = reinterpret_cast<unsigned long long*>(result_dev);
  best_ij = best_d2 + nslots;
  best_f32 = reinterpret_cast<float*>(best_ij + nslots);
  seed_bsf = reinterpret_cast<unsigned int*>(best_f32 + nslots);
  Q.counters = reinterpret_cast<unsigned long long*>(result_dev + at_counters);
  Q.cand_count = reinterpret_cast<unsigned int*>(Q.counters + kNumCounters);
  status_dev = reinterpret_cast<int*>(Q.cand_count + 1);

  // every buffer of the call in one allocation, the group filter's and the
  // window table's only where they fit the device
  DevSeries S;
  PrepScratch P;
  // search state
  unsigned int qcap = kQueueCapMax;
  if (const char* env = getenv("DTWJ_QUEUE_CAP")) {  // smaller queue (profiling, tests)
    const long v = atol(env);
    if (v >= 1024 && v < (long)kQueueCapMax) qcap = (unsigned int)v;
  }
  const bool enumerate_all = flags & DTWJ_F_NO_DIAG;
  const double full_tile = (double)kLbLags * kLbRows;
  int chunk = ctx->chunk_tiles > 0 ? ctx->chunk_tiles
                                   : kLbChunkRounds * kLbCtasPerSm * ctx->num_sms;
  if (enumerate_all) chunk = (int)((double)qcap / full_tile) > 0 ? (int)((double)qcap / full_tile) : 1;
  const int chunk_max = chunk < nlb ? chunk : (nlb > 0 ? nlb : 1);  // tiles of the largest chunk
  // LB_Keogh candidates of one chunk, and those that go on to DTW (nearly all
  // of them on quasi-periodic series): no more than the call has pairs
  double pairs_bound = 1024.0;
  for (int r = 0; r < nseries; ++r) {
    const double k = (double)((sbeg ? sbeg[r + 1] - sbeg[r] : n) - 2 * (int64_t)m + 1);
    pairs_bound += 0.5 * k * (k + 1.0);
  }
  const unsigned int queue_cap =
      pairs_bound < 2.0 * qcap ? (unsigned int)pairs_bound : qcap * 2;
  Q.queue_cap = Q.kq_cap = queue_cap;
  // the tile minima keep a few candidates per tile
  const unsigned int cand_cap =
      tile_mode && 16u * (unsigned int)nlb > kCandCap ? 16u * (unsigned int)nlb : kCandCap;
  Q.cand_cap = cand_cap;
  using Range = std::pair<int, int>;
  std::vector<Range> ranges;
  for (int t0 = 0; t0 < nlb; t0 += chunk) ranges.push_back({t0, t0 + chunk < nlb ? t0 + chunk : nlb});
  const bool want_features = learned || (tq && tq->features);
  const bool want_keys = nlb > 0 && (tile_mode || want_features || !(flags & DTWJ_F_NO_SEED));
  // counters of a chunk, then the group filter's surviving group pairs per tile
  constexpr int kQcTiles = 16;
  unsigned int *qc, *nseeds, *bits, *probe;  // nseeds: [nseries] counts, total slots, work counter
  unsigned long long* keys;          // row minima of the ED profile
  int2* seeds;
  ChunkNote* notes;
  double* vd2;
  GroupFilter F;
  memset(&F, 0, sizeof F);
  const size_t table = 3 * (size_t)(n - m + 1) * ((m + 3) / 4 * 4) * sizeof(float);
  bool want_table = band.C <= 8 && table <= kWindowTableMax && !(tq && !tile_mode);
  Prep level = enumerate_all || (tq && !tile_mode) ? kPrepSweep : kPrepJoin;
  int rc = DTWJ_OK;
  for (;;) {
    Arena A;
    plan_series(A, x_dev, n, m, w, masked, level, sbeg, nseries, &S, &P);
    if (want_keys) A.add(&keys, S.s * 8);
    if (!tq || tile_mode) {
      A.add(&qc, (size_t)(kQcTiles + chunk_max) * 4);
      A.add(&F.dense, (size_t)chunk_max * 4);
      A.add(&Q.bsf2, (size_t)nslots * 4);
      A.add(&S.zready, 8);
      A.add(&Q.low, 8);
      A.add(&probe, 8);
      A.add(&seeds, (size_t)nseries * kSeedSlots * sizeof(int2));
      A.add(&nseeds, ((size_t)nseries + 2) * 4);
      A.add(&notes, (ranges.size() + 1) * sizeof(ChunkNote));
      A.add(&Q.cand, (size_t)cand_cap * sizeof(Candidate));
      A.add(&vd2, (size_t)cand_cap * 8);
      if (level == kPrepJoin && m <= (1 << kBlkShift)) {
        const size_t pairs = (size_t)chunk_max * group_items(S.grp_g, &F);
        A.add(&F.sup, pairs * 4);
        A.add(&F.list, pairs * sizeof(uint2));
        F.sup_cap = F.list_cap = (unsigned int)pairs;
      }
      A.add(&bits, (size_t)chunk_max * kLbLags * kLbWords * 4);
      if (tile_mode) A.add(&Q.qser, (size_t)queue_cap * sizeof(int));
      if (want_table) A.add(&S.zt, table);
      A.add(&Q.queue, (size_t)queue_cap * sizeof(int2));
      A.add(&Q.kq, (size_t)queue_cap * sizeof(int4));
    }
    rc = A.place(ctx, B_WORK);
    if (rc != DTWJ_ERR_OOM) break;
    if (want_table) want_table = false;
    else if (level == kPrepJoin) level = kPrepSweep;
    else break;
  }
  if (rc) return rc;
  S.status = status_dev;
  if (want_table) {
    S.zm = (m + 3) / 4 * 4;
    S.zu = S.zt + S.s * S.zm;
    S.zl = S.zu + S.s * S.zm;
  }
  rc = prepare(ctx, S, P, &ph);
  if (rc) return rc;
  S.nseries = nslots;
  if (tile_mode)
    for (int t = 0; t < nlb; ++t) th[t].series = t;
  Tile* lbtiles;
  ENSURE(B_LBTILES, (size_t)(nlb > 0 ? nlb : 1) * sizeof(Tile), lbtiles);
  if (!keep_tiles) {
    if (nlb > 0)
      CUDA_OK(cudaMemcpyAsync(lbtiles, th.data(), (size_t)nlb * sizeof(Tile),
                              cudaMemcpyHostToDevice, st));
    ctx->tiles_dev = {sbeg || tile_mode ? nullptr : lbtiles, n, m, rank, world};
  }

  unsigned int *lb_next = nullptr, *paa_next = nullptr;
  if (!tq || tile_mode) {
    Q.queue_count = qc;
    Q.queue_next = qc + 1;
    Q.run_count = qc + 2;
    Q.run_next = qc + 3;
    Q.kq_count = qc + 4;
    Q.kq_next = qc + 5;
    lb_next = qc + 6;
    F.nsup = qc + 8;
    F.nlist = qc + 9;
    F.ndense = qc + 10;
    paa_next = qc + 11;
    if (S.grp) F.tcount = qc + kQcTiles;
    k_init_search<<<(nslots + 255) / 256 < 256 ? (nslots + 255) / 256 : 256, 256, 0, st>>>(
        Q.bsf2, nslots, Q.counters, Q.cand_count, nseeds, nseries, nseries * kSeedSlots, S.zready,
        Q.low, probe);
    if (S.grp && nlb >= kProbeTiles) F.probe = probe;
  }

  // ---- ED matrix profile (row minima; per tile for the tile minima) ----
  if (want_keys) {
    unsigned int* tbest = nullptr;
    if (tile_mode) {
      ENSURE(B_TILEBEST, (size_t)nlb * 4, tbest);
      CUDA_OK(cudaMemsetAsync(tbest, 0xff, (size_t)nlb * 4, st));
    }
    ph.begin();
    // a join only ranks seed candidates by these keys (mixed precision, one
    // row in kSeedGrid); the per-tile minima and the exported features take
    // the exact FP64 profile of every row
    int launches = 2;
    if (tq) {
      launch_mp(S, lbtiles, nlb, keys, st, tbest);
    } else if (S.grp && !sbeg && !learned && nlb >= kSeedGroupTiles &&
               (size_t)chunk_max * kLbLags * kLbWords * 4 >= kSeedScratch) {
      // a large join: the group bound finds the rows; its lists lie in the
      // survivor bits' buffer, which the sweep uses later
      GroupFilter E = F;
      E.sup_cap = kSeedSupCap;
      E.list_cap = kSeedListCap;
      E.sup = bits;
      E.list = reinterpret_cast<uint2*>(bits + kSeedSupCap);
      float* samples = reinterpret_cast<float*>(E.list + kSeedListCap);
      unsigned int* word = reinterpret_cast<unsigned int*>(samples + kSeedSamples);
      E.nsup = word;
      E.nlist = word + 1;
      E.tcount = word + 2;
      E.walk = word + 3;
      E.probe = word + 4;
      E.cut = reinterpret_cast<const float*>(word + 6);
      launch_seed_groups(S, E, lbtiles, nlb, ctx->shard_world, samples, keys, ctx->num_sms, st);
      launch_mp_seed(S, lbtiles, nlb, keys, E.walk, ctx->num_sms, st);
      launches = 4 + 3 * ((nlb + kSeedSlab - 1) / kSeedSlab);
    } else {
      launch_mp_seed(S, lbtiles, nlb, keys, nullptr, ctx->num_sms, st);
      launches = 1;
    }
    if (tile_mode) launch_tile_bound(tbest, nlb, Q.bsf2, st);
    ph.end(DTWJ_PHASE_PROFILE, launches);
  }
  // ---- tile features; the learned order sorts the tiles by their score ----
  if (want_features && nlb > 0) {
    float* feat;
    ENSURE(B_FEAT, (size_t)nlb * DTWJ_MLP_IN * 4, feat);
    launch_tile_features(S, lbtiles, nlb, keys, tq ? 1 : kSeedGrid, feat, st);
    if (tq && tq->features)
      CUDA_OK(cudaMemcpyAsync(tq->features, feat, (size_t)nlb * DTWJ_MLP_IN * 4,
                              cudaMemcpyDeviceToHost, st));
    if (learned) {
      float* score;
      ENSURE(B_SCORE, (size_t)nlb * 4, score);
      rc = mlp_predict_device(ctx->model, feat, nlb, score, st);
      if (rc) return rc;
      // ascending predicted minimum; ties (and NaN scores, last) keep the
      // plain order: a stable radix sort of (score key, tile) on the device,
      // then the tiles gathered in that order
      unsigned int* sk;
      ENSURE(B_SORT, (size_t)nlb * 16, sk);
      unsigned int* sk_out = sk + nlb;
      int* si = reinterpret_cast<int*>(sk + 2 * (size_t)nlb);
      int* si_out = si + nlb;
      const unsigned int nb = (unsigned int)((nlb + 255) / 256);
      k_order_keys<<<nb, 256, 0, st>>>(score, nlb, sk, si);
      size_t temp_bytes = 0;
      CUDA_OK(cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, sk, sk_out, si, si_out, nlb,
                                              0, 32, st));
      void* temp;
      ENSURE(B_SORT_TEMP, temp_bytes > 0 ? temp_bytes : 16, temp);
      CUDA_OK(cub::DeviceRadixSort::SortPairs(temp, temp_bytes, sk, sk_out, si, si_out, nlb, 0,
                                              32, st));
      Tile* sorted;
      ENSURE(B_LBTILES2, (size_t)nlb * sizeof(Tile), sorted);
      k_gather_tiles<<<nb, 256, 0, st>>>(lbtiles, si_out, nlb, sorted);
      lbtiles = sorted;
    }
  }
  if (tq && !tile_mode) {
    CUDA_OK(cudaStreamSynchronize(st));
    return DTWJ_OK;
  }

  // ---- ED profile seeds ----
  if (!tile_mode && !(flags & DTWJ_F_NO_SEED) && nlb > 0) {
    ph.begin();
    launch_seed_select(S, keys, seeds, nseeds, st);
    DevSearch Qs = Q;
    Qs.qser = nullptr;
    Qs.queue_next = nseeds + nseries + 1;
    Qs.queue_cap = (unsigned int)(nseries * kSeedSlots);
    launch_pairs(S, Qs, seeds, nseeds + nseries, false, wide, ctx->num_sms, st);
    if (F.probe) launch_group_probe(S, Q, F, lbtiles, nlb, st);
    ph.end(DTWJ_PHASE_SEEDS, F.probe ? 3 : 2);
  }
  CUDA_OK(cudaMemcpyAsync(seed_bsf, Q.bsf2, (size_t)nslots * 4, cudaMemcpyDeviceToDevice, st));

  // ---- diagonal sweep in chunks of LB tiles ----
  // the stages after the diagonal bound of one chunk: run filter, LB_Keogh, DTW
  auto filter_chunk = [&](int t0, int t1) {
    ph.begin();
    if (enumerate_all || cascade) {
      launch_runs(S, Q, lbtiles, t0, t1, bits, masked, !enumerate_all, ctx->num_sms, st);
      ph.end(DTWJ_PHASE_RUNS, 1);
    } else {
      if (S.grp) launch_paa_groups(S, Q, F, lbtiles, t0, t1, paa_next, ctx->num_sms, st);
      launch_paa(S, Q, F, lbtiles, t0, t1, bits, ctx->num_sms, st);
      ph.end(DTWJ_PHASE_RUNS, S.grp ? 2 : 1);
    }
    if (!enumerate_all) {
      ph.begin();
      launch_keogh(S, Q, ctx->num_sms, st);
      if (petitjean) launch_petitjean(S, Q, qc + 7, ctx->num_sms, st);
      ph.end(DTWJ_PHASE_KEOGH, petitjean ? 2 : 1);
    }
    ph.begin();
    if (S.zt) launch_window_table(S, Q, ctx->num_sms, st);
    launch_pairs(S, Q, Q.queue, Q.queue_count, true, band, ctx->num_sms, st);
    ph.end(DTWJ_PHASE_PAIRS, S.zt ? 2 : 1);
  };
  // one pass over tile ranges: bound sweep, run filter, LB_Keogh, DTW, and a
  // note of each range (queue overflow, counters after it); notes[0] holds
  // the counters before the pass, notes[c + 1] those after range c
  auto sweep_range = [&](const Range& r, ChunkNote* note) {
    CUDA_OK(cudaMemsetAsync(qc, 0, (size_t)(kQcTiles + r.second - r.first) * 4, st));
    ph.begin();
    if (S.grp) launch_group(S, Q, F, lbtiles, r.first, r.second, ctx->num_sms, st);
    launch_lb(S, Q, F, lbtiles, r.first, r.second, bits, enumerate_all, cascade, lb_next,
              ctx->num_sms, st);
    if (S.grp && cascade)
      launch_group_bits(S, Q, F, lbtiles, r.first, ctx->num_sms, bits, st);
    ph.end(DTWJ_PHASE_DIAG, S.grp ? (cascade ? 4 : 3) : 1);
    filter_chunk(r.first, r.second);
    k_chunk_note<<<1, 32, 0, st>>>(S.status, Q.counters, note);
    return DTWJ_OK;
  };
  auto sweep = [&](const std::vector<Range>& rg, ChunkNote* notes) -> int {
    k_chunk_note<<<1, 32, 0, st>>>(S.status, Q.counters, notes);
    for (size_t c = 0; c < rg.size(); ++c) sweep_range(rg[c], notes + c + 1);
    CUDA_OK(cudaGetLastError());
    return DTWJ_OK;
  };
  // a sharded join with an exchange sweeps its tiles in phases and lets the
  // caller lower the best-so-far between them (direct launches)
  const bool exchanging = ctx->exchange && ctx->shard_world > 1 && !tq;
  auto sweep_phased = [&]() -> int {
    const int P = ctx->exchange_phases;
    k_chunk_note<<<1, 32, 0, st>>>(S.status, Q.counters, notes);
    size_t c = 0;
    for (int ph_i = 0; ph_i < P; ++ph_i) {
      const int b = (int)((int64_t)nlb * (ph_i + 1) / P);
      for (; c < ranges.size() && ranges[c].second <= b; ++c)
        sweep_range(ranges[c], notes + c + 1);
      ctx->exchange(ctx->exchange_user, Q.bsf2, nslots, (void*)st);
    }
    for (; c < ranges.size(); ++c) sweep_range(ranges[c], notes + c + 1);
    CUDA_OK(cudaGetLastError());
    return DTWJ_OK;
  };
  // FP64 verification of the candidates, the minimum per series, and the
  // result block on its way to the host
  unsigned char* result = staging(ctx, result_bytes);
  auto finish = [&]() -> int {
    ph.begin();
    launch_verify(S, Q, wide, vd2, best_d2, best_ij, best_f32, st);
    ph.end(DTWJ_PHASE_VERIFY, 4);
    CUDA_OK(cudaGetLastError());
    CUDA_OK(cudaEventRecord(ctx->ev1, st));
    CUDA_OK(cudaMemcpyAsync(result, result_dev, result_bytes, cudaMemcpyDeviceToHost, st));
    CUDA_OK(cudaStreamSynchronize(st));
    return DTWJ_OK;
  };
  const int* status_h = reinterpret_cast<const int*>(result + at_counters + kNumCounters * 8 + 4);
  // A batch sweeps chunk by chunk and checks each one: its short series put
  // many tiles' survivors into one chunk, and when a chunk's queues
  // overflow, the counters go back to before it, it is swept again in
  // chunks an eighth its size, and the size grows back after chunks that
  // fit, up to half the size that overflowed (a pass that is checked only at
  // its end would sweep every overflowing chunk twice).
  const bool adaptive = sbeg != nullptr && !exchanging && nlb > 0;
  if (adaptive) {
    ChunkNote* an;
    ENSURE(B_NOTES2, 2 * sizeof(ChunkNote), an);
    k_chunk_note<<<1, 32, 0, st>>>(S.status, Q.counters, an);
    int ch = chunk, ch_max = chunk;
    size_t resweeps = 0;
    for (int t0 = 0; t0 < nlb;) {
      const int t1 = t0 + ch < nlb ? t0 + ch : nlb;
      sweep_range({t0, t1}, an + 1);
      ChunkNote h[2];
      CUDA_OK(cudaMemcpyAsync(h, an, sizeof h, cudaMemcpyDeviceToHost, st));
      CUDA_OK(cudaStreamSynchronize(st));
      if (!h[1].overflow) {
        CUDA_OK(cudaMemcpyAsync(an, an + 1, sizeof(ChunkNote), cudaMemcpyDeviceToDevice, st));
        t0 = t1;
        ch = 2 * ch < ch_max ? 2 * ch : ch_max;
        continue;
      }
      if (t1 - t0 == 1) return DTWJ_ERR_OVERFLOW;
      ++resweeps;
      CUDA_OK(cudaMemcpyAsync(Q.counters, h[0].counters, sizeof h[0].counters,
                              cudaMemcpyHostToDevice, st));
      CUDA_OK(cudaStreamSynchronize(st));  // h is read before it goes out of scope
      ch_max = (t1 - t0) / 2 > 0 ? (t1 - t0) / 2 : 1;
      ch = (t1 - t0) / 8 > 0 ? (t1 - t0) / 8 : 1;
    }
    CUDA_OK(cudaGetLastError());
    if (verbose && resweeps)
      fprintf(stderr, "dtwj: %zu chunks swept again in smaller chunks\n", resweeps);
    if ((rc = finish())) return rc;
  }
  for (int attempt = 0; !adaptive; ++attempt) {
    bool swept = false;
    ChunkNote* pass_notes = notes;
    // only the first pass exchanges: a shard whose queues overflowed sweeps
    // those chunks again alone, and every shard must make the same exchange
    // calls
    if (exchanging && attempt == 0) {
      const int src = sweep_phased();
      if (src) return src;
      swept = true;
    }
    if (!swept && attempt == 0 && !(flags & DTWJ_F_NO_GRAPH) && nlb > 0) {
      // the first pass runs as a CUDA graph: replayed if this context captured
      // the same launches before, captured (then launched) otherwise
      std::vector<unsigned char> key;
      auto put = [&key](const void* p, size_t bytes) {
        const unsigned char* b = static_cast<const unsigned char*>(p);
        key.insert(key.end(), b, b + bytes);
      };
      const int band_cg[3] = {band.C, band.G, band.warps};
      const int64_t misc[12] = {nlb, chunk, enumerate_all, masked, cascade, petitjean,
                                ctx->num_sms, ph.on,
                                (int64_t)ph.used, (int64_t)(uintptr_t)lbtiles,
                                (int64_t)(uintptr_t)bits, (int64_t)(uintptr_t)notes};
      put(&S, sizeof S);
      put(&Q, sizeof Q);
      put(&F, sizeof F);
      put(band_cg, sizeof band_cg);
      put(misc, sizeof misc);
      // a context's first join launches directly: it may be its only one
      const bool seen = key == ctx->sweep_seen;
      if (!seen) ctx->sweep_seen = key;
      if (ctx->sweep_exec && key == ctx->sweep_key) {
        CUDA_OK(cudaGraphLaunch(ctx->sweep_exec, st));
        for (size_t k = 0; k + 3 < ctx->sweep_marks.size(); k += 4)
          ph.marks.push_back({ctx->sweep_marks[k], (size_t)ctx->sweep_marks[k + 1],
                              (size_t)ctx->sweep_marks[k + 2], ctx->sweep_marks[k + 3]});
        ph.used = ctx->sweep_ev1;
        swept = true;
      } else if (seen) {
        if (ctx->sweep_exec) cudaGraphExecDestroy(ctx->sweep_exec);
        ctx->sweep_exec = nullptr;
        ctx->sweep_key.clear();
        const size_t u0 = ph.used, m0 = ph.marks.size();
        // events the capture records must exist before it starts
        if (ph.on) ph.ev(u0 + 8 * ranges.size() + 8);
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        bool ok = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
        if (ok) {
          ph.capturing = true;
          const int src = sweep(ranges, notes);
          ph.capturing = false;
          ok = cudaStreamEndCapture(st, &graph) == cudaSuccess && src == DTWJ_OK && graph;
        }
        if (ok) ok = cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
        if (graph) cudaGraphDestroy(graph);
        if (ok && cudaGraphLaunch(exec, st) == cudaSuccess) {
          ctx->sweep_exec = exec;
          ctx->sweep_key = key;
          ctx->sweep_marks.clear();
          for (size_t k = m0; k < ph.marks.size(); ++k) {
            const auto& mk = ph.marks[k];
            ctx->sweep_marks.insert(ctx->sweep_marks.end(),
                                    {mk.phase, (int)mk.a, (int)mk.b, mk.launches});
          }
          ctx->sweep_ev0 = u0;
          ctx->sweep_ev1 = ph.used;
          swept = true;
        } else {
          // not capturable here: fall back to direct launches
          if (exec) cudaGraphExecDestroy(exec);
          cudaGetLastError();
          ph.used = u0;
          ph.marks.resize(m0);
        }
      }
    }
    if (!swept) {
      if (attempt > 0) {
        // the chunks swept again get notes of their own (the first pass's
        // buffer stays as the captured graph knows it)
        ENSURE(B_NOTES2, (ranges.size() + 1) * sizeof(ChunkNote), pass_notes);
      }
      const int src = sweep(ranges, pass_notes);
      if (src) return src;
    }
    if ((rc = finish())) return rc;
    // a chunk whose queue overflowed lost pairs: take its counts out and
    // sweep it again in smaller chunks (the other chunks stand)
    if (ranges.empty() || !(*status_h & kOverflowSeen)) break;
    CUDA_OK(cudaMemsetAsync(S.status, 0, 4, st));
    std::vector<ChunkNote> nh(ranges.size() + 1);
    CUDA_OK(cudaMemcpyAsync(nh.data(), pass_notes, nh.size() * sizeof(ChunkNote),
                            cudaMemcpyDeviceToHost, st));
    CUDA_OK(cudaStreamSynchronize(st));
    std::vector<Range> again;
    unsigned long long drop[kNumCounters] = {0};
    size_t nbad = 0;
    for (size_t c = 0; c < ranges.size(); ++c) {
      if (!nh[c + 1].overflow) continue;
      ++nbad;
      for (int k = 0; k < kNumCounters; ++k)
        drop[k] += nh[c + 1].counters[k] - nh[c].counters[k];
      const int t0 = ranges[c].first, t1 = ranges[c].second;
      if (t1 - t0 == 1 || attempt >= 4) return DTWJ_ERR_OVERFLOW;
      int sub = (t1 - t0) / 32;
      if (sub > kResweepTiles) sub = kResweepTiles;
      if (sub < 1) sub = 1;
      for (int u = t0; u < t1; u += sub) again.push_back({u, u + sub < t1 ? u + sub : t1});
    }
    if (again.empty()) break;
    if (verbose)
      fprintf(stderr, "dtwj: queue overflow in %zu of %zu chunks, sweeping them again in %zu\n",
              nbad, ranges.size(), again.size());
    unsigned long long kept[kNumCounters];
    for (int k = 0; k < kNumCounters; ++k) kept[k] = nh.back().counters[k] - drop[k];
    CUDA_OK(cudaMemcpyAsync(Q.counters, kept, sizeof kept, cudaMemcpyHostToDevice, st));
    CUDA_OK(cudaStreamSynchronize(st));  // kept is read before it goes out of scope
    ranges.swap(again);
  }

  // ---- results ----
  const unsigned long long* d2_h = reinterpret_cast<const unsigned long long*>(result);
  const unsigned long long* ij_h = d2_h + nslots;
  const unsigned int* f32_h = reinterpret_cast<const unsigned int*>(ij_h + nslots);
  const unsigned int* seed_h = f32_h + nslots;
  const unsigned long long* cnt_h =
      reinterpret_cast<const unsigned long long*>(result + at_counters);
  const unsigned int cand_h = *reinterpret_cast<const unsigned int*>(cnt_h + kNumCounters);
  if (*status_h & 2) return DTWJ_ERR_OVERFLOW;
  if (cand_h > cand_cap) return DTWJ_ERR_OVERFLOW;
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  if (tile_mode) {
    for (int t = 0; t < nlb; ++t) {
      double d2;
      memcpy(&d2, &d2_h[t], 8);
      tq->min_dist[t] = d2_h[t] != ~0ull ? std::sqrt(d2) : INFINITY;
    }
    return DTWJ_OK;
  }

  for (int r = 0; r < nseries; ++r) {
    dtwj_result* out = &outs[r];
    memset(out, 0, sizeof *out);
    const int64_t base = sbeg ? sbeg[r] : 0;
    out->n = sbeg ? sbeg[r + 1] - sbeg[r] : n;
    out->m = m;
    out->w = w_in;
    if (d2_h[r] != ~0ull) {
      double d2;
      memcpy(&d2, &d2_h[r], 8);
      float f2;
      memcpy(&f2, &f32_h[r], 4);
      out->i = (int64_t)(ij_h[r] >> 32) - base;
      out->j = (int64_t)(ij_h[r] & 0xffffffffull) - base;
      out->dist = std::sqrt(d2);
      out->dist_fp32 = std::sqrt((double)f2);
    } else {
      out->i = out->j = -1;
      out->dist = out->dist_fp32 = INFINITY;
    }
    float sb;
    memcpy(&sb, &seed_h[r], 4);
    out->seed_bsf = std::sqrt((double)sb);
    out->seconds_join = ms / 1000.0;
    out->seconds_total = wall.seconds() + t_upload;
    if (!sbeg) {  // the counters are the whole call's: per series only for a single join
      out->pairs = cnt_h[kPairs];
      out->pruned_fast = cnt_h[kPrunedFast];
      out->pruned_kim = cnt_h[kPrunedKim];
      out->pruned_masked = cnt_h[kPrunedMasked];
      out->pruned_keogh = cnt_h[kPrunedKeogh];
      out->pruned_paa = cnt_h[kPrunedPaa];
      out->pruned_petitjean = cnt_h[kPrunedPetitjean];
      out->dtw_calls = cnt_h[kDtwCalls];
      out->dtw_abandoned = cnt_h[kDtwAbandoned];
      out->dtw_cells = cnt_h[kDtwCells];
      out->candidates = cand_h;
      ph.collect(out);
    }
  }
  if (verbose)
    fprintf(stderr, "dtwj: %d series, %.3fs device, %u candidates\n", nseries, ms / 1000.0, cand_h);
  return DTWJ_OK;
}

int join_device(dtwj_ctx* ctx, const double* x_dev, int64_t n, int32_t m, int32_t w_in,
                uint32_t flags, dtwj_result* out, double t_upload) {
  return run_join(ctx, x_dev, n, nullptr, 1, m, w_in, flags, out, t_upload);
}

int upload(dtwj_ctx* ctx, const double* x, int64_t n, double** dev) {
  ENSURE(B_A, n * 8, *dev);
  CUDA_OK(cudaMemcpyAsync(*dev, x, n * 8, cudaMemcpyHostToDevice, ctx->stream));
  return DTWJ_OK;
}

}  // namespace

extern "C" {

int dtwj_device_count(void) {
  int c = 0;
  if (cudaGetDeviceCount(&c) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return c;
}

int dtwj_ctx_create(int device, dtwj_ctx** out) {
  if (!out) return DTWJ_ERR_ARG;
  *out = nullptr;
  if (dtwj_device_count() <= device || device < 0) return DTWJ_ERR_NODEVICE;
  dtwj_ctx* c = new (std::nothrow) dtwj_ctx();
  if (!c) return DTWJ_ERR_OOM;
  c->device = device;
  if (cudaSetDevice(device) != cudaSuccess) {
    delete c;
    return DTWJ_ERR_CUDA;
  }
  cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess) {
    cudaGetLastError();
    c->bufs.resize(B_COUNT_);
    dtwj_ctx_destroy(c);
    return DTWJ_ERR_CUDA;
  }
  c->bufs.resize(B_COUNT_);
  *out = c;
  return DTWJ_OK;
}

void dtwj_ctx_destroy(dtwj_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  for (auto& b : c->bufs)
    if (b.p) cudaFree(b.p);
  if (c->sweep_exec) cudaGraphExecDestroy(c->sweep_exec);
  for (auto e : c->pool) cudaEventDestroy(e);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

int dtwj_ctx_join_device(dtwj_ctx* ctx, const double* x_dev, int64_t n, int32_t m, int32_t w,
                         uint32_t flags, dtwj_result* out) {
  if (!ctx || !out) return DTWJ_ERR_ARG;
  int rc = check_args(x_dev, n, m, w);
  if (rc) return rc;
  cudaSetDevice(ctx->device);
  return join_device(ctx, x_dev, n, m, w, flags, out, 0.0);
}

int dtwj_band_shapes(int32_t w, int32_t* C, int32_t* G, int32_t max) {
  if (w < 0 || max < 0 || (max > 0 && (!C || !G))) return DTWJ_ERR_ARG;
  BandShape b[16];
  const int k = band_shapes(w, b, 16);
  for (int q = 0; q < k && q < max && q < 16; ++q) {
    C[q] = b[q].C;
    G[q] = b[q].G;
  }
  return k;
}

int dtwj_ctx_set_band(dtwj_ctx* ctx, int32_t w, int32_t C, int32_t G) {
  if (!ctx || w < 0) return DTWJ_ERR_ARG;
  auto& v = ctx->band_override;
  for (size_t q = 0; q < v.size(); ++q)
    if (v[q].first == w) {
      v.erase(v.begin() + q);
      break;
    }
  if (C == 0 && G == 0) return DTWJ_OK;
  if (!band_shape_ok(w, C, G)) return DTWJ_ERR_BAND;
  v.push_back({w, BandShape{C, G}});
  return DTWJ_OK;
}

int dtwj_ctx_set_tuning(dtwj_ctx* ctx, int32_t dtw_warps, int32_t chunk_tiles) {
  if (!ctx) return DTWJ_ERR_ARG;
  if (dtw_warps != 0 && dtw_warps != 1 && dtw_warps != 2 && dtw_warps != 4 && dtw_warps != 8)
    return DTWJ_ERR_ARG;
  if (chunk_tiles != 0 && (chunk_tiles < 16 || chunk_tiles > 4096)) return DTWJ_ERR_ARG;
  ctx->dtw_warps = dtw_warps;
  ctx->chunk_tiles = chunk_tiles;
  return DTWJ_OK;
}

int dtwj_time_band(int device, int32_t m, int32_t w, int32_t C, int32_t G, int32_t pairs,
                   double* cells_per_s) {
  if (!cells_per_s || m < 8 || m > DTWJ_MAX_M || w < 0 || pairs < 1) return DTWJ_ERR_ARG;
  const int we = effective_band(m, w);
  if (!band_shape_ok(we, C, G)) return DTWJ_ERR_BAND;
  dtwj_ctx* ctx = nullptr;
  int rc = dtwj_ctx_create(device, &ctx);
  if (rc) return rc;
  do {
    // a seeded random walk of 8m samples, pairs of windows drawn from it
    const int64_t n = 8 * (int64_t)m;
    std::vector<double> x((size_t)n);
    uint64_t st = 0x9e3779b97f4a7c15ull;
    double v = 0.0;
    for (int64_t p = 0; p < n; ++p) {
      st = st * 6364136223846793005ull + 1442695040888963407ull;
      v += ((double)(st >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
      x[(size_t)p] = v;
    }
    double* dev = nullptr;
    if ((rc = upload(ctx, x.data(), n, &dev))) break;
    DevSeries S;
    PrepScratch P;
    if ((rc = plan_and_prepare(ctx, dev, n, m, we, false, kPrepStats, &S, &P))) break;
    std::vector<int2> pr((size_t)pairs);
    const int64_t s = n - m + 1;
    for (int q = 0; q < pairs; ++q) {
      st = st * 6364136223846793005ull + 1442695040888963407ull;
      const int a = (int)((st >> 33) % (uint64_t)(s - m));
      st = st * 6364136223846793005ull + 1442695040888963407ull;
      const int b = a + m + (int)((st >> 33) % (uint64_t)(s - m - a));
      pr[(size_t)q] = make_int2(a, b);
    }
    int2* dp;
    double* out;
    if ((rc = ensure(ctx, B_PAIRS, (size_t)pairs * sizeof(int2), (void**)&dp))) break;
    if ((rc = ensure(ctx, B_OUT, (size_t)pairs * 8, (void**)&out))) break;
    if (cudaMemcpyAsync(dp, pr.data(), (size_t)pairs * sizeof(int2), cudaMemcpyHostToDevice,
                        ctx->stream) != cudaSuccess) {
      rc = DTWJ_ERR_CUDA;
      break;
    }
    const BandShape b = {C, G};
    launch_pair_dtw(S, dp, pairs, false, b, out, ctx->stream);  // warm-up
    cudaEventRecord(ctx->ev0, ctx->stream);
    for (int r = 0; r < 3; ++r) launch_pair_dtw(S, dp, pairs, false, b, out, ctx->stream);
    cudaEventRecord(ctx->ev1, ctx->stream);
    if (cudaStreamSynchronize(ctx->stream) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
      rc = DTWJ_ERR_CUDA;
      break;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    const double cells = 3.0 * pairs * ((double)m * (2 * we + 1) - (double)we * (we + 1));
    *cells_per_s = ms > 0 ? cells / (ms * 1e-3) : 0.0;
  } while (0);
  dtwj_ctx_destroy(ctx);
  return rc;
}

int dtwj_ctx_set_shard(dtwj_ctx* ctx, int32_t rank, int32_t world) {
  if (!ctx || world < 1 || rank < 0 || rank >= world) return DTWJ_ERR_ARG;
  ctx->shard_rank = rank;
  ctx->shard_world = world;
  return DTWJ_OK;
}

int dtwj_ctx_set_exchange(dtwj_ctx* ctx, dtwj_exchange_fn fn, void* user, int32_t phases) {
  if (!ctx || (fn && phases < 1)) return DTWJ_ERR_ARG;
  ctx->exchange = fn;
  ctx->exchange_user = fn ? user : nullptr;
  ctx->exchange_phases = fn ? phases : 0;
  return DTWJ_OK;
}

int dtwj_ctx_set_model(dtwj_ctx* ctx, dtwj_mlp* net) {
  if (!ctx) return DTWJ_ERR_ARG;
  if (net && mlp_device(net) != ctx->device) return DTWJ_ERR_ARG;
  ctx->model = net;
  return DTWJ_OK;
}

int dtwj_ctx_tiles(dtwj_ctx* ctx, const double* x, int64_t n, int32_t m, int32_t w,
                   int64_t* count, int32_t* desc, float* features, double* min_dist) {
  if (!ctx || !count) return DTWJ_ERR_ARG;
  int rc = check_args(x, n, m, w);
  if (rc) return rc;
  cudaSetDevice(ctx->device);
  build_lb_tiles(ctx, n, m, nullptr, 1);
  const int64_t nt = (int64_t)ctx->lbtiles_host.size();
  *count = nt;
  if (desc) {
    const int64_t s = n - m + 1;
    for (int64_t t = 0; t < nt; ++t) {
      const Tile& T = ctx->lbtiles_host[t];
      const int64_t lags = s - T.i0 - T.L0 < kLbLags ? s - T.i0 - T.L0 : kLbLags;
      desc[4 * t] = T.L0;
      desc[4 * t + 1] = T.i0;
      desc[4 * t + 2] = T.rows;
      desc[4 * t + 3] = (int32_t)lags;
    }
  }
  if (!features && !min_dist) return DTWJ_OK;
  double* dev = nullptr;
  rc = upload(ctx, x, n, &dev);
  if (rc) return rc;
  TileQuery tq;
  tq.features = features;
  tq.min_dist = min_dist;
  if (min_dist && features) {
    // features first (a plain pass), then the minima sweep
    TileQuery f1 = {features, nullptr};
    rc = run_join(ctx, dev, n, nullptr, 1, m, w, 0, nullptr, 0.0, &f1);
    if (rc) return rc;
    tq.features = nullptr;
  }
  return run_join(ctx, dev, n, nullptr, 1, m, w, DTWJ_F_NO_GRAPH, nullptr, 0.0, &tq);
}

int dtwj_ctx_join(dtwj_ctx* ctx, const double* x, int64_t n, int32_t m, int32_t w,
                  uint32_t flags, dtwj_result* out) {
  if (!ctx || !out) return DTWJ_ERR_ARG;
  int rc = check_args(x, n, m, w);
  if (rc) return rc;
  cudaSetDevice(ctx->device);
  Timer t;
  double* dev = nullptr;
  rc = upload(ctx, x, n, &dev);
  if (rc) return rc;
  rc = join_device(ctx, dev, n, m, w, flags, out, 0.0);
  if (rc == DTWJ_OK) out->seconds_total = t.seconds();
  return rc;
}

int dtwj_join(const double* x, int64_t n, int32_t m, int32_t w, uint32_t flags,
              dtwj_result* out) {
  if (!out) return DTWJ_ERR_ARG;
  int rc = check_args(x, n, m, w);
  if (rc) return rc;
  dtwj_ctx* ctx = nullptr;
  rc = dtwj_ctx_create(0, &ctx);
  if (rc) return rc;
  rc = dtwj_ctx_join(ctx, x, n, m, w, flags, out);
  dtwj_ctx_destroy(ctx);
  return rc;
}

int dtwj_join_batch(const double* const* xs, const int64_t* ns, const int32_t* ms,
                    const int32_t* ws, int32_t count, uint32_t flags, dtwj_result* outs) {
  if (!xs || !ns || !ms || !ws || !outs || count < 0) return DTWJ_ERR_ARG;
  int rc = DTWJ_OK;
  for (int32_t k = 0; k < count && rc == DTWJ_OK; ++k) rc = check_args(xs[k], ns[k], ms[k], ws[k]);
  if (rc || count == 0) return rc;
  // series of one (m, effective band) are joined together, back to back
  std::vector<int32_t> order(count);
  for (int32_t k = 0; k < count; ++k) order[k] = k;
  auto key = [&](int32_t k) {
    return ((int64_t)ms[k] << 32) | (uint32_t)effective_band(ms[k], ws[k]);
  };
  std::stable_sort(order.begin(), order.end(),
                   [&](int32_t a, int32_t b) { return key(a) < key(b); });
  std::vector<std::pair<int32_t, int32_t>> groups;  // [g0, g1) of order
  for (int32_t g0 = 0; g0 < count;) {
    int32_t g1 = g0;
    while (g1 < count && key(order[g1]) == key(order[g0])) ++g1;
    groups.push_back({g0, g1});
    g0 = g1;
  }
  // One group's pass on a context: its series stored back to back, joined
  // together, each result written to its own slot of outs.
  auto run_group = [&](dtwj_ctx* ctx, int32_t g0, int32_t g1, std::vector<double>& cat,
                       std::vector<int64_t>& sbeg, std::vector<dtwj_result>& res) -> int {
    const int nser = g1 - g0;
    sbeg.assign(1, 0);
    for (int32_t q = g0; q < g1; ++q) sbeg.push_back(sbeg.back() + ns[order[q]]);
    const int64_t total = sbeg.back();
    if (total > (int64_t)INT32_MAX - 4) return DTWJ_ERR_ARG;
    cat.resize((size_t)total);
    for (int32_t q = g0; q < g1; ++q)
      memcpy(cat.data() + sbeg[q - g0], xs[order[q]], (size_t)ns[order[q]] * 8);
    double* dev = nullptr;
    Timer t;
    int grc = upload(ctx, cat.data(), total, &dev);
    if (grc) return grc;
    res.resize((size_t)nser);
    grc = run_join(ctx, dev, total, sbeg.data(), nser, ms[order[g0]], ws[order[g0]], flags,
                   res.data(), 0.0);
    for (int q = 0; q < nser && grc == DTWJ_OK; ++q) {
      res[q].w = ws[order[g0 + q]];
      res[q].seconds_total = t.seconds();
      outs[order[g0 + q]] = res[q];
    }
    return grc;
  };
  // Groups run concurrently, up to kBatchWorkers at a time: each worker
  // thread owns a context (its own stream and buffers) and takes the next
  // group until none is left, so one group's host checks and small launches
  // overlap another's kernels.
  const int workers = (int)groups.size() < kBatchWorkers ? (int)groups.size() : kBatchWorkers;
  std::atomic<int> next_group{0};
  std::atomic<int> first_error{DTWJ_OK};
  auto worker = [&]() {
    dtwj_ctx* ctx = nullptr;
    int wrc = dtwj_ctx_create(0, &ctx);
    std::vector<double> cat;
    std::vector<int64_t> sbeg;
    std::vector<dtwj_result> res;
    while (wrc == DTWJ_OK && first_error.load() == DTWJ_OK) {
      const int gi = next_group.fetch_add(1);
      if (gi >= (int)groups.size()) break;
      wrc = run_group(ctx, groups[gi].first, groups[gi].second, cat, sbeg, res);
    }
    if (wrc != DTWJ_OK) {
      int expected = DTWJ_OK;
      first_error.compare_exchange_strong(expected, wrc);
    }
    dtwj_ctx_destroy(ctx);
  };
  std::vector<std::thread> pool;
  if (workers > 1) {
    try {
      for (int k = 0; k < workers; ++k) pool.emplace_back(worker);
    } catch (...) {
      // no more threads: the workers already started take every group
    }
  }
  if (pool.empty()) worker();
  for (auto& th : pool) th.join();
  return first_error.load();
}

int dtwj_matrix_profile(const double* x, int64_t n, int32_t m, double* mp, int64_t* mpi) {
  if (!mp || !mpi) return DTWJ_ERR_ARG;
  int rc = check_args(x, n, m, 0);
  if (rc) return rc;
  dtwj_ctx* ctx = nullptr;
  rc = dtwj_ctx_create(0, &ctx);
  if (rc) return rc;
  do {
    double* dev = nullptr;
    if ((rc = upload(ctx, x, n, &dev))) break;
    build_lb_tiles(ctx, n, m, nullptr, 1);
    const int nlb = (int)ctx->lbtiles_host.size();
    const int64_t s = n - m + 1;
    const unsigned int cap =
        (unsigned int)(s * 16 + 4096 < (1ll << 31) ? s * 16 + 4096 : (1ll << 31));
    DevSeries S;
    PrepScratch P;
    Tile* tiles;
    double* dmp;
    int64_t* dmpi;
    unsigned long long *rowmin, *rowidx;
    unsigned int *best, *cnt;
    int2 *cand_up, *cand_lo;
    Arena A;
    plan_series(A, dev, n, m, 0, false, kPrepProfile, nullptr, 1, &S, &P);
    A.add(&tiles, (size_t)nlb * sizeof(Tile));
    A.add(&dmp, s * 8);
    A.add(&dmpi, s * 8);
    A.add(&rowmin, s * 8);
    A.add(&rowidx, s * 8);
    A.add(&best, s * 4);
    A.add(&cnt, 8);
    A.add(&cand_up, (size_t)cap * sizeof(int2));
    A.add(&cand_lo, (size_t)cap * sizeof(int2));
    if ((rc = A.place(ctx, B_WORK))) break;
    if ((rc = prepare(ctx, S, P))) break;
    cudaStream_t st = ctx->stream;
    cudaMemcpyAsync(tiles, ctx->lbtiles_host.data(), (size_t)nlb * sizeof(Tile),
                    cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(best, 0xff, s * 4, st);
    cudaMemsetAsync(cnt, 0, 8, st);
    cudaMemsetAsync(rowmin, 0xff, s * 8, st);
    cudaMemsetAsync(rowidx, 0xff, s * 8, st);
    // The first walk keeps the high word of ED^2 per window; every pair near it
    // (near_limit, mp.cu) for either of its windows is a candidate, its FP64
    // distance is computed directly, and the row takes the smallest, lowest
    // partner on ties.
    launch_profile(S, tiles, nlb, false, best, nullptr, nullptr, nullptr, 0, ctx->num_sms,
                   st);
    launch_profile(S, tiles, nlb, true, best, cand_up, cand_lo, cnt, cap, ctx->num_sms,
                   st);
    for (int pick = 0; pick < 2; ++pick) {
      launch_mp_exact(S, cand_up, cnt, cap, pick != 0, rowmin, rowidx, st);
      launch_mp_exact(S, cand_lo, cnt + 1, cap, pick != 0, rowmin, rowidx, st);
    }
    launch_mp_exact_out(s, rowmin, rowidx, dmp, dmpi, st);
    unsigned int cnt_h[2] = {0, 0};
    if (cudaMemcpyAsync(cnt_h, cnt, 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      rc = DTWJ_ERR_CUDA;
      break;
    }
    if (cnt_h[0] > cap || cnt_h[1] > cap) {
      // more ties than the lists hold (a periodic series): again, a few tiles at
      // a time, with lists that hold every pair of them
      constexpr int kSlab = 8;
      constexpr size_t kSlabPairs = (size_t)kSlab * kLbLags * kLbRows;
      void* p;
      if ((rc = ensure(ctx, B_OUT, 2 * kSlabPairs * sizeof(int2), &p))) break;
      cand_up = static_cast<int2*>(p);
      cand_lo = cand_up + kSlabPairs;
      cudaMemsetAsync(rowmin, 0xff, s * 8, st);
      cudaMemsetAsync(rowidx, 0xff, s * 8, st);
      for (int pick = 0; pick < 2; ++pick)
        for (int t = 0; t < nlb; t += kSlab) {
          const int k = nlb - t < kSlab ? nlb - t : kSlab;
          cudaMemsetAsync(cnt, 0, 8, st);
          launch_profile(S, tiles + t, k, true, best, cand_up, cand_lo, cnt,
                         (unsigned int)kSlabPairs, ctx->num_sms, st);
          launch_mp_exact(S, cand_up, cnt, (unsigned int)kSlabPairs, pick != 0, rowmin, rowidx, st);
          launch_mp_exact(S, cand_lo, cnt + 1, (unsigned int)kSlabPairs, pick != 0, rowmin, rowidx,
                          st);
        }
      launch_mp_exact_out(s, rowmin, rowidx, dmp, dmpi, st);
    }
    if (cudaMemcpyAsync(mp, dmp, s * 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(mpi, dmpi, s * 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      rc = DTWJ_ERR_CUDA;
      break;
    }
  } while (0);
  dtwj_ctx_destroy(ctx);
  return rc;
}

int dtwj_global_mask(const double* x, int64_t n, int32_t m, int32_t w, float* mask,
                     int32_t* table_len) {
  if (!mask) return DTWJ_ERR_ARG;
  int rc = check_args(x, n, m, w);
  if (rc) return rc;
  const int we = effective_band(m, w);
  dtwj_ctx* ctx = nullptr;
  rc = dtwj_ctx_create(0, &ctx);
  if (rc) return rc;
  do {
    double* dev = nullptr;
    if ((rc = upload(ctx, x, n, &dev))) break;
    DevSeries S;
    PrepScratch P;
    if ((rc = plan_and_prepare(ctx, dev, n, m, we, true, kPrepSweep, &S, &P))) break;
    if (cudaMemcpyAsync(mask, S.mask, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
      rc = DTWJ_ERR_CUDA;
      break;
    }
    if (table_len) {
      // the table length the mask used: 200 floor(max |z|), at least 600
      float zmax = 0.0f;
      if (cudaMemcpy(&zmax, P.zmax, 4, cudaMemcpyDeviceToHost) != cudaSuccess) {
        rc = DTWJ_ERR_CUDA;
        break;
      }
      const int lt = (int)(std::floor((double)zmax) * 200.0);
      *table_len = lt > 600 ? lt : 600;
    }
  } while (0);
  dtwj_ctx_destroy(ctx);
  return rc;
}

int dtwj_pair_dtw(const double* x, int64_t n, int32_t m, int32_t w, const int64_t* pi,
                  const int64_t* pj, int64_t count, int32_t precise, double* dist) {
  if (!pi || !pj || !dist || count < 0) return DTWJ_ERR_ARG;
  int rc = check_args(x, n, m, w);
  if (rc) return rc;
  const int64_t s = n - m + 1;
  std::vector<int2> pairs((size_t)count);
  for (int64_t k = 0; k < count; ++k) {
    if (pi[k] < 0 || pj[k] < 0 || pi[k] >= s || pj[k] >= s) return DTWJ_ERR_ARG;
    pairs[k] = make_int2((int)pi[k], (int)pj[k]);
  }
  if (count == 0) return DTWJ_OK;
  const int we = effective_band(m, w);
  BandShape band;
  if (!choose_band(we, &band)) return DTWJ_ERR_BAND;
  if (!choose_band_pairs(m, we, count, precise != 0, &band)) return DTWJ_ERR_ARG;
  dtwj_ctx* ctx = nullptr;
  rc = dtwj_ctx_create(0, &ctx);
  if (rc) return rc;
  do {
    double* dev = nullptr;
    if ((rc = upload(ctx, x, n, &dev))) break;
    DevSeries S;
    PrepScratch P;
    if ((rc = plan_and_prepare(ctx, dev, n, m, we, false, kPrepStats, &S, &P))) break;
    void* p;
    if ((rc = ensure(ctx, B_PAIRS, (size_t)count * sizeof(int2), &p))) break;
    int2* dp = (int2*)p;
    if ((rc = ensure(ctx, B_OUT, (size_t)count * 8, &p))) break;
    double* dout = (double*)p;
    cudaMemcpyAsync(dp, pairs.data(), (size_t)count * sizeof(int2), cudaMemcpyHostToDevice,
                    ctx->stream);
    launch_pair_dtw(S, dp, (int)count, precise != 0, band, dout, ctx->stream);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(dist, dout, (size_t)count * 8, cudaMemcpyDeviceToHost, ctx->stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
      rc = DTWJ_ERR_CUDA;
      break;
    }
    for (int64_t k = 0; k < count; ++k) dist[k] = std::sqrt(dist[k]);
  } while (0);
  dtwj_ctx_destroy(ctx);
  return rc;
}

int dtwj_pair_lb_petitjean(const double* x, int64_t n, int32_t m, int32_t w, const int64_t* pa,
                           const int64_t* pb, int64_t count, int32_t own_env, double* keogh_mid,
                           double* terms) {
  if (!pa || !pb || !keogh_mid || !terms || count < 0 || count > INT32_MAX) return DTWJ_ERR_ARG;
  int rc = check_args(x, n, m, w);
  if (rc) return rc;
  const int we = effective_band(m, w);
  if (lbp_list_bytes(m, we, own_env != 0) > kPjMaxSmemBytes) return DTWJ_ERR_ARG;
  const int64_t s = n - m + 1;
  std::vector<int2> pairs((size_t)count);
  for (int64_t k = 0; k < count; ++k) {
    if (pa[k] < 0 || pb[k] < 0 || pa[k] >= s || pb[k] >= s) return DTWJ_ERR_ARG;
    pairs[k] = make_int2((int)pa[k], (int)pb[k]);
  }
  if (count == 0) return DTWJ_OK;
  dtwj_ctx* ctx = nullptr;
  rc = dtwj_ctx_create(0, &ctx);
  if (rc) return rc;
  do {
    double* dev = nullptr;
    if ((rc = upload(ctx, x, n, &dev))) break;
    DevSeries S;
    PrepScratch P;
    if ((rc = plan_and_prepare(ctx, dev, n, m, we, false, kPrepSweep, &S, &P))) break;
    void* p;
    if ((rc = ensure(ctx, B_PAIRS, (size_t)count * sizeof(int2), &p))) break;
    int2* dp = (int2*)p;
    if ((rc = ensure(ctx, B_OUT, (size_t)count * 16, &p))) break;
    double* dout = (double*)p;
    cudaMemcpyAsync(dp, pairs.data(), (size_t)count * sizeof(int2), cudaMemcpyHostToDevice,
                    ctx->stream);
    launch_lbp_list(S, dp, (int)count, own_env != 0, dout, dout + count, ctx->num_sms,
                    ctx->stream);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(keogh_mid, dout, (size_t)count * 8, cudaMemcpyDeviceToHost,
                        ctx->stream) != cudaSuccess ||
        cudaMemcpyAsync(terms, dout + count, (size_t)count * 8, cudaMemcpyDeviceToHost,
                        ctx->stream) != cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
      rc = DTWJ_ERR_CUDA;
      break;
    }
  } while (0);
  dtwj_ctx_destroy(ctx);
  return rc;
}

int32_t dtwj_band(int32_t m, double ratio, int32_t rounding) {
  double v = ratio * (double)m;
  int32_t w;
  if (rounding == 1) w = (int32_t)std::floor(v + 0.5);
  else w = (int32_t)std::ceil(v - 1e-9);
  return w < 1 ? 1 : w;
}

const char* dtwj_strerror(int code) {
  switch (code) {
    case DTWJ_OK: return "ok";
    case DTWJ_ERR_ARG: return "invalid argument";
    case DTWJ_ERR_NAN: return "input contains NaN or infinity";
    case DTWJ_ERR_CUDA: return "CUDA error";
    case DTWJ_ERR_OOM: return "device out of memory";
    case DTWJ_ERR_BAND: return "band too wide (w must be <= 255)";
    case DTWJ_ERR_OVERFLOW: return "candidate or survivor list overflow";
    case DTWJ_ERR_TIMEOUT: return "device-side wait ran out";
    case DTWJ_ERR_NODEVICE: return "no CUDA device";
    case DTWJ_ERR_IO: return "file could not be read or written";
    case DTWJ_ERR_NOMODEL: return "learned ordering requested but no model is loaded";
    case DTWJ_ERR_SCRATCH: return "series exceeds the fixed scratch of the allocation-free entry point";
    default: return "unknown error";
  }
}

}  // extern "C"
