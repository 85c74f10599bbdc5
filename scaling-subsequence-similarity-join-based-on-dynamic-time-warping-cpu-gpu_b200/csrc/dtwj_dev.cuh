// Internal header: device-side layout of one prepared series and the launch
// entry points of every kernel of the join.  Host orchestration (join.cu)
// only sees the launch functions declared at the bottom.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace dtwj {

// Relative slack on squared distances for every pruning and abandoning test.
// FP32 distances and the FP64 diagonal recurrences carry rounding error far
// below this; the slack keeps every pair whose true distance can still be the
// minimum, and the final candidates are re-verified in FP64.
constexpr float kSlack = 1.0f / 512.0f;
// Absolute slack per window sample on squared distances: keeps a pair whose
// distance ties the best-so-far (exact duplicates give 0) above the rounding
// of the FP32 bounds.
constexpr float kAbsSlackPerSample = 1e-6f;

// Pruning / abandoning threshold on squared distances from the best-so-far.
__device__ __forceinline__ float prune_threshold(unsigned int bsf2_bits, int m) {
  return __uint_as_float(bsf2_bits) * (1.0f + kSlack) + kAbsSlackPerSample * (float)m;
}
__device__ __forceinline__ float prune_threshold_now(const unsigned int* bsf2, int m) {
  return prune_threshold(*(volatile const unsigned int*)bsf2, m);
}

// Whether an FP32 lower bound built from block-centered copies (LB_Keogh,
// the block-mean bound) may prune a pair whose windows have error scale r
// (the larger of their DevSeries::rw), against the squared threshold thr.
// Every z-like difference such a bound forms is within dz = 16 * 2^-24 * r of
// its exact value (the centered value, the FP32 reciprocal deviation, the
// block offset and each FMA round once, every term bounded by a few r), so a
// bound sum_k c_k d_k^2 with sum_k c_k <= m is within
// 2 dz sqrt(m * bound) + m dz^2 of the exact one at bound <= thr, plus the
// FP32 summation (at most m / 8 + 8 terms per lane, relative 2^-24 each).
// The pair may be pruned when that error fits in the slack thr keeps above
// the best-so-far: thr - bsf2 = (thr kSlack + kAbsSlackPerSample m) / (1 + kSlack).
__device__ __forceinline__ bool fp32_bound_ok(float r, float thr, int m) {
  const float fm = (float)m;
  const float dz = r * (16.0f / 16777216.0f);
  const float err = 2.0f * dz * sqrtf(fm * thr) + fm * dz * dz +
                    thr * ((fm * 0.125f + 8.0f) * (1.0f / 16777216.0f));
  const float slack = (thr * kSlack + kAbsSlackPerSample * fm) * (1.0f / (1.0f + kSlack));
  return err <= slack;
}

// The largest error scale r for which fp32_bound_ok(r, thr, m) holds (the
// error bound is increasing in r): the positive root of
// a r^2 + b r + c = 0 with a = m k^2, b = 2 k sqrt(m thr), c = summation term
// - slack, k = 16 * 2^-24, in the form -2c / (b + sqrt(b^2 - 4ac)) that does
// not cancel, shrunk by 2^-10 against the rounding of this evaluation; -1 if
// none.
__device__ __forceinline__ float fp32_bound_radius(float thr, int m) {
  const float fm = (float)m, k = 16.0f / 16777216.0f;
  const float slack = (thr * kSlack + kAbsSlackPerSample * fm) * (1.0f / (1.0f + kSlack));
  const float c = thr * ((fm * 0.125f + 8.0f) * (1.0f / 16777216.0f)) - slack;
  if (!(c < 0.0f)) return -1.0f;  // also +inf / NaN thresholds: no FP32 pruning
  const float a = fm * k * k, b = 2.0f * k * sqrtf(fm * thr);
  const float r = -2.0f * c / (b + sqrtf(b * b - 4.0f * a * c));
  return r * (1.0f - 1.0f / 1024.0f);
}

// Endpoint bound width (the reference's BIAS, CPU_version1/diag_mask_global.cpp:8).
constexpr int kBias = 3;
// Seeds taken from the ED matrix profile (CPU_version1/new_dtw_motifGUI.cpp:53).
constexpr int kSeeds = 100;
// The seed profile keys one row in kSeedGrid; each seed pair is widened to
// kSeedSpread pairs on its diagonal (offsets -kSeedGrid/2 .. kSeedGrid/2).
constexpr int kSeedGrid = 7;
constexpr int kSeedSpread = kSeedGrid;
constexpr int kSeedSlots = kSeeds * kSeedSpread;
// Sentinels padding the z-normalised sequences: finite so that no
// inf - inf appears, far enough apart that any cell touching them is
// effectively infinite.
constexpr float kPadQ = 1e18f;
constexpr float kPadT = -1e18f;
constexpr double kPadQd = 1e150;
constexpr double kPadTd = -1e150;

// Lag-block x row-block of the diagonal sweep: pairs (i, i + L) for
// L in [L0, L0 + kLbLags) and i in [i0, i0 + rows), all windows below send.
// Indices are global: in a batch the series sit back to back and a tile
// belongs to one of them.
struct Tile {
  int32_t L0;
  int32_t i0;
  int32_t rows;
  int32_t order;   // position in the queue order (learned or plain)
  int32_t send;    // end of the series' windows (global window index)
  int32_t series;  // series of the batch (0 for a single join)
};
// Diagonal-sweep tiles: 128 threads x kLbPerThread lags x kLbRows rows, one
// survivor bit per pair, kLbWords 32-row words per lag.
constexpr int kLbThreads = 128;
constexpr int kLbPerThread = 7;
constexpr int kLbLags = kLbThreads * kLbPerThread;
constexpr int kLbRows = 18 * kLbPerThread * 32;
constexpr int kLbWords = kLbRows / 32;
// CTAs of the persistent diagonal sweep per SM (launch bounds of k_lb).
constexpr int kLbCtasPerSm = 3;
// Lags per group of the block-mean filter's work items (one lag per lane).
constexpr int kLbGroups = kLbLags / 32;
static_assert(kLbLags % 32 == 0, "lag groups of one warp");
// Longest run of consecutive surviving rows the sweep emits as one item.
constexpr int kRunMax = 256;
// FP32 copies of the series and its envelopes are centered per block of
// 2^kBlkShift samples (value minus the block mean) so that the float rounding
// error stays far below the pruning slack.
constexpr int kBlkShift = 10;
// Blocks of each copy of DevSeries::pq2 (copy 1's block b starts 1024
// samples before copy 0's).
__host__ __device__ inline int64_t kCopyBlocks(int64_t n) { return (n >> 11) + 2; }

// Counters, all uint64 on the device.
enum Counter {
  kPairs = 0,
  kPrunedFast,
  kPrunedKim,
  kPrunedMasked,
  kPrunedKeogh,
  kDtwCalls,
  kDtwAbandoned,
  kDtwCells,
  kCandidates,
  kPrunedPaa,
  kPrunedPetitjean,
  kNumCounters
};

struct Candidate {
  int32_t i, j;
  float d2;
  int32_t series;
};

// All device arrays of one prepared series.
struct DevSeries {
  const double* a;  // n, the series (a batch: all series back to back)
  int64_t n;
  int64_t s;        // n - m + 1
  int m, w;
  const int* sid;   // n, series of each sample (nullptr for a single series)
  const int64_t* sbeg;  // series + 1 sample offsets (nullptr for a single series)
  int nseries;
  double* mu;       // s, window mean
  double* sig;      // s, window population std (1 for flat windows)
  double* isg;      // s, 1/sig (0 for flat windows)
  uint8_t* flat;    // s
  double* U;        // n, upper envelope of the raw series, radius w
  double* L;        // n, lower envelope
  double* E;        // n, U + L
  double* nu;       // s, mean of (U + L) over the window
  double* dfa;      // s, (a[i+m] - a[i]) / 2
  double* dga;      // s, (a[i+m] - mu[i+1]) + (a[i] - mu[i])
  double* dfE;      // s, same for E = U + L
  double* dgE;      // s
  double* A;        // s, 4m + 2N - DUL2   (fast bound row constant)
  double* DUL;      // s, ||nU - nL||
  double* qsig;     // s, sig / 4 (1e300-guarded for flat windows)
  float* mask;      // n, 0/1 mask of the masked bound
  float* MN;        // s, sum_T M (nU^2 + nL^2)
  float* MDUL2;     // s, sum_m M (nU - nL)^2
  float* MDUL;      // s
  double* SM;       // s, sum_T M            (T = [kBias, m-1-kBias])
  double* SME;      // s, sum_T M (E - 2 mu)
  double* cb;       // (n >> kBlkShift) + 2, block centers
  float* af;        // n, a - cb[block]
  float2* ulf;      // n, (U - cb[block], L - cb[block])
  int paa_b;        // block length of the block-mean bound (8, 16 or 32)
  float4* pq;       // n, means over [p, p + paa_b) of (a, U, L) - cb[block of p], 0
                    //    (windows longer than 1024 samples; else nullptr)
  float* cmax;      // (n >> kBlkShift) + 2, largest |centered FP32 value| per block
  float* rw;        // s, FP32 error scale of window i: isg_i x the largest
                    //    centered magnitude or block offset its FP32 bounds read
  // Windows of at most 1024 samples: the same block means in two copies
  // centered per 2048-sample block, copy 0 on [2048 b, 2048 b + 2048) and
  // copy 1 on [2048 b - 1024, 2048 b + 1024), so every window lies inside one
  // block of one copy and has a single block offset (else all nullptr).
  float4* pq2;      // 2n, copy c at [c n, c n + n)
  float* fq;        // the same over fine blocks of paa_b / 4 samples, a apart from
  float2* ful;      //    (U, L) and phase-major (fine_at): a window's blocks are consecutive
  int64_t fine_n;   // entries per phase
  float* cmax2;     // 2 kCopyBlocks(n), largest |value| of each copy block (both lengths)
  float4* wrec;     // s, window record: block offset (FP64 in .x/.y), isg as
                    //    FP32 (.z) and the error scale for pq2 (.w)
  // Window groups of the group bound (nullptr: not built): grp_d slots of
  // grp_n records, slot-major; a record holds (smallest and largest block
  // mean, largest upper and smallest lower envelope mean) of grp_g windows
  // over one segment of grp_b samples, z-normalised, rounded outward.
  float4* grp;
  float4* sup;      // the same for kGrpFan consecutive groups, sup_n records per slot
  int64_t grp_n, sup_n;
  int grp_g, grp_b, grp_d;
  // Window table of the DTW stage (nullptr: too large): the z-normalised
  // windows and their envelopes as FP32 rows of zm values, filled by
  // launch_window_table once a chunk queues enough pairs (*zready).
  float *zt, *zu, *zl;
  int zm;
  unsigned int* zready;  // [0] filled, [1] blocks done
  int* status;      // device status word (0 ok, else error bits)
};

// The copy whose blocks hold window [i, i + m), m <= 1024: copy 0 when the
// window ends inside its 2048-sample block, else copy 1 (then i mod 2048 >
// 1024 and the window lies in [2048 b + 1024, 2048 b + 3072)).
__device__ __forceinline__ int win_copy(int64_t i, int m) { return (int)(i & 2047) + m > 2048 ? 1 : 0; }
// Fine block [p, p + F) of copy c, F = paa_b / 4; the next block of the same
// window, at p + F, follows it.
__device__ __forceinline__ int64_t fine_at(const DevSeries& S, int c, int64_t p) {
  const int F = S.paa_b / 4;
  return ((int64_t)c * F + p % F) * S.fine_n + p / F;
}

// Global search state of one join.
struct DevSearch {
  unsigned int* bsf2;           // per series: float bits of the best squared DTW so far
  unsigned long long* counters; // kNumCounters
  Candidate* cand;              // candidate list
  unsigned int* cand_count;
  unsigned int cand_cap;
  int4* runs;                   // runs of fast-bound survivors: (i0, j0, len, 0)
  unsigned int* run_count;
  unsigned int* run_next;
  unsigned int run_cap;
  int2* queue;                  // survivor pairs of the current chunk
  int* qser;                    // their best-so-far slot (nullptr: the series of i)
  unsigned int* queue_count;
  unsigned int* queue_next;
  unsigned int queue_cap;
  int4* kq;                     // LB_Keogh candidates: (query, envelope, endpoint bound bits,
                                //   series), the more promising direction first
  unsigned int* kq_count;
  unsigned int* kq_next;
  unsigned int kq_cap;
  unsigned int* low;            // [2] of this join: of the pairs well below the threshold, those
                                //   LB_Keogh tried and counted, and those of them it pruned
};

__device__ __forceinline__ float max3f(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// ---- group filter (group.cu) ----
constexpr int kGrpSlots = 32;  // segments per window, at most
constexpr int kGrpFan = 4;     // groups of a super-group
// Windows per group.  A group's records widen with the shift between its
// windows, which matters relative to m: of a random walk's pairs, groups of 8
// and 4 let through 1.8 % and 1.0 % at m = 512, w = 52 (single pairs: 0.7 %),
// 0.64 % and 0.11 % at m = 256, w = 13 (0.02 %), 6.6 % and 1.9 % at m = 128.
__host__ __device__ inline int group_windows(int m) { return m >= 512 ? 8 : 4; }
// Buffers of the filter over one chunk of tiles.
struct GroupFilter {
  unsigned int* sup;     // surviving super-group pairs: group_code
  unsigned int* nsup;
  uint2* list;           // of them, those with surviving group pairs: (group_code, mask of the
                         //   kGrpFan x kGrpFan group pairs)
  unsigned int* nlist;
  unsigned int* tcount;  // surviving group pairs per tile (nullptr: no filter, every tile dense)
  unsigned int sup_cap, list_cap;
  const float* cut;      // seeds only: the cutoff on ED^2 ...
  unsigned int* walk;    // ... and whether the diagonals must be walked after all
  unsigned int* probe;   // [2] sampled group pairs, those that survive (nullptr: none sampled)
  unsigned int* dense;   // tiles the diagonal sweep ran on
  unsigned int* ndense;
  int nib, nw;           // first-level work items per tile: blocks of row groups x column words
};
// Whether the bound settles too little to be worth its time on this join (every
// tile is dense then): by the sample, more than one in `den` survivors of ED
// pairs, 15/16 of the sweep's (a tile stays sparse at 7/8 or less, so hardly any
// would).
__device__ __forceinline__ bool group_off(const GroupFilter& F, bool ed, unsigned int den) {
  if (!F.probe) return false;
  return ed ? F.probe[1] * den > F.probe[0] : F.probe[1] * 16u > F.probe[0] * 15u;
}
// One group pair in 128 (g = 8) or 256 may survive a seed's cutoff (k_seed_exact's
// budget); twice that in a sample is too many.
__device__ __forceinline__ unsigned int seed_share(int g) { return g == 8 ? 64u : 128u; }
// A super-group pair of a tile of the chunk: tile, row group relative to the
// tile's first (at most 252), column group relative to row group + L0 / G (at
// most 57).
__host__ __device__ inline unsigned int group_code(unsigned int tile, int row, int col) {
  return (tile << 14) | ((unsigned int)row << 6) | (unsigned int)col;
}
__host__ __device__ inline unsigned int group_code_tile(unsigned int code) { return code >> 14; }
struct GroupPair {
  int I, J;
};
__host__ __device__ inline GroupPair group_code_pair(unsigned int code, const Tile& T, int G) {
  GroupPair p;
  p.I = T.i0 / G + (int)((code >> 6) & 255u);
  p.J = p.I + T.L0 / G + (int)(code & 63u);
  return p;
}
// Whether a pair of groups of g windows holds pairs of the tile (for groups
// that reach past the tile's rows or lags on both sides: may hold).
__host__ __device__ inline bool group_pair_in_tile(const Tile& T, int g, int I, int J) {
  const int64_t ia = (int64_t)I * g, ja = (int64_t)J * g, last = (int64_t)T.i0 + T.rows - 1;
  const int64_t lo = ia > T.i0 ? ia : T.i0, hi = ia + g - 1 < last ? ia + g - 1 : last;
  return lo <= hi && ja < T.send && ja + g - 1 - lo >= T.L0 && ja - hi < T.L0 + kLbLags;
}
// Pairs of a tile: rows [0, rows), lags [0, kLbLags) with the later window
// below send.
__host__ __device__ inline int64_t tile_pairs(const Tile& T) {
  const int64_t room = (int64_t)T.send - T.i0 - T.L0;  // lags of the first row, >= rows
  int64_t full = room - kLbLags + 1;                   // rows with every lag
  full = full < 0 ? 0 : (full < T.rows ? full : T.rows);
  const int64_t part = T.rows - full;
  return full * kLbLags + part * (room - full) - part * (part - 1) / 2;
}
// A tile goes through the diagonal bound when more than 7/8 of its group
// pairs survive: the group bound says nothing about it (noise, or structure
// shorter than a segment), where the diagonal bound may still prune.
__host__ __device__ inline bool group_tile_dense(const Tile& T, int g, unsigned int count) {
  return (int64_t)count * g * g * 8 > 7 * tile_pairs(T);
}

// Endpoint bound: minimum cost of any warping path's cells in the first and
// last three layers (LB_KIM, CPU_version1/lb_kim.cpp:10-73).  q = window i,
// t = window j (any indexable sequences); cells are (t index, q index).  The
// reference's fourth option adds the corner cell twice (lb_kim.cpp:55,62);
// here it is added once so that the bound stays admissible.
template <typename V, typename Seq>
__device__ __forceinline__ V kim_side(const Seq& q, const Seq& t) {
  auto D2 = [](V x, V y) { return (x - y) * (x - y); };
  auto mn = [](V x, V y) { return x < y ? x : y; };
  const V o = D2(t[0], q[0]);
  const V lw = mn(D2(t[1], q[0]), D2(t[1], q[1]));
  const V l1 = mn(lw, D2(t[0], q[1]));
  V d = mn(D2(t[1], q[0]) + D2(t[2], q[0]), lw + D2(t[2], q[1]));
  d = mn(d, D2(q[1], t[1]) + D2(q[2], t[2]));
  d = mn(d, l1 + D2(q[2], t[1]));
  d = mn(d, D2(q[1], t[0]) + D2(q[2], t[0]));
  return o + d;
}
template <typename Seq>
struct Reversed {
  const Seq& s;
  int e;
  __device__ auto operator[](int k) const { return s[e - k]; }
};
// left from the windows' first three samples, right from their last three.
template <typename V, typename Seq>
__device__ __forceinline__ void kim_bound(const Seq& q, const Seq& t, int m, V* left, V* right) {
  *left = kim_side<V>(q, t);
  *right = kim_side<V>(Reversed<Seq>{q, m - 1}, Reversed<Seq>{t, m - 1});
}

struct BandShape {
  int C;  // cells (diagonals) per lane
  int G;  // lanes per pair
  int warps = 0;  // CTA size of the join's DTW kernel in warps (0: the default, 2 in slots, else 4)
};
// One pair per warp (G = 32) with the fewest cells per lane C in [2, 16]
// covering 2w+1 diagonals.  Returns false if w > 255.
bool choose_band(int w, BandShape* out);
// The join's layout: several pairs to a warp where the band and the windows
// are small enough, else choose_band.
bool choose_band_join(int m, int w, BandShape* out);
// Exact DTW lists (no early abandoning): G in {4, 8, 16, 32} and C in
// [2, 16] covering 2w+1 diagonals with the least waste.
bool choose_band_list(int w, BandShape* out);
// Whether a list of pairs in this layout runs: the windows of a warp's pairs
// lie in shared memory.
bool pair_list_fits(int m, BandShape band, bool precise);
// The layout of a list of `count` pairs; false: w > 255 or none fits.
bool choose_band_pairs(int m, int w, int64_t count, bool precise, BandShape* out);
// (C, G) has a kernel instantiation and covers band w.
bool band_shape_ok(int w, int C, int G);
// The shapes the autotuner tries for band w (per G the two smallest covering
// C); writes up to max, returns how many there are.
int band_shapes(int w, BandShape* out, int max);

// ---- launches (all on `stream`) ----
void launch_check_finite(const double* a, int64_t n, int* status, cudaStream_t st);
// sid[p] = series of sample p for a batch with series offsets sbeg[0..nseries].
void launch_series_ids(const int64_t* sbeg, int nseries, int* sid, int64_t n, cudaStream_t st);
void launch_prep(const DevSeries& S, cudaStream_t st);
void launch_stats(const DevSeries& S, cudaStream_t st);
// Update terms of the series alone (dfa, dga); returns the kernels launched.
int launch_diffs(const DevSeries& S, cudaStream_t st);
void launch_rowterms(const DevSeries& S, bool masked, cudaStream_t st);
// Largest CDF length the mask can need: max |z| <= sqrt(m - 1).
int mask_table_max(int m);
void launch_mask(const DevSeries& S, unsigned int* counts, int lt_max, double* diff,
                 double* mean_acc, float* zmax, cudaStream_t st);
// Row minima over partners j >= i + m on LB tiles (lb.cu layout).
// With tile_best (ntiles entries, 0xffffffff at launch): also each tile's
// smallest key high bits.
void launch_mp(const DevSeries& S, const Tile* tiles, int ntiles, unsigned long long* keys,
               cudaStream_t st, unsigned int* tile_best = nullptr);
// bsf2[t] = an upper bound on tile t's smallest squared DTW (its ED^2 minimum).
void launch_tile_bound(const unsigned int* tile_best, int ntiles, unsigned int* bsf2,
                       cudaStream_t st);
// Matrix profile: best[i] = the smallest high word of ED^2 over window i's
// partners on both sides (collect = false; best starts at 0xffffffff); then
// (collect = true) the pairs near it, as (row, later partner) in up and (row,
// earlier partner) in lo, count[2] how many there are.  The exact pass computes
// the FP64 distance of such a list (pick = false: row minima of the bits, true:
// lowest partner at the minimum).
void launch_profile(const DevSeries& S, const Tile* tiles, int ntiles, bool collect,
                    unsigned int* best, int2* up, int2* lo, unsigned int* count, unsigned int cap,
                    int num_sms, cudaStream_t st);
void launch_mp_exact(const DevSeries& S, const int2* cand, const unsigned int* count,
                     unsigned int cap, bool pick, unsigned long long* rowmin,
                     unsigned long long* rowidx, cudaStream_t st);
void launch_mp_exact_out(int64_t s, const unsigned long long* rowmin,
                         const unsigned long long* rowidx, double* mp, int64_t* mpi,
                         cudaStream_t st);
// kSeeds seeds per series, each with its diagonal neighbours, into
// seeds[series * kSeedSlots ...] (unused slots hold (-1, -1)), their counts
// into nseeds[series].
void launch_seed_select(const DevSeries& S, const unsigned long long* keys, int2* seeds,
                        unsigned int* nseeds, cudaStream_t st);
// Row minima for the join's seeds on the rows of a kSeedGrid grid: FP64
// anchors and stage carries, FP32 increments within a stage (keys only rank
// the seed candidates).
// walk (nullptr: always): the kernel returns at once while *walk is zero, and
// adds to the keys instead of starting from empty ones.
void launch_mp_seed(const DevSeries& S, const Tile* tiles, int ntiles, unsigned long long* keys,
                    const unsigned int* walk, int num_sms, cudaStream_t st);
// The same keys for the rows that can be among the kSeeds smallest, by the
// group bound (group.cu).  F: lists of sup_cap and list_cap entries, nsup,
// nlist, tcount (one word: the group pair count) consecutive, walk and probe
// consecutive, cut; samples: kSeedSamples floats.  Single series.
constexpr int kSeedSamples = 2048;
constexpr int kSeedSlab = 16384;  // tiles per pass
void launch_seed_groups(const DevSeries& S, GroupFilter F, const Tile* tiles, int ntiles,
                        int world, float* samples, unsigned long long* keys, int num_sms,
                        cudaStream_t st);
// Series of a sample (0 for a single series).
__device__ __forceinline__ int series_of(const DevSeries& S, int64_t x) {
  return S.sid ? S.sid[x] : 0;
}
// Group filter (group.cu).  group_shape sets the group sizes of S;
// launch_group_prep fills S.grp and S.sup (means: 3 n doubles of scratch) and
// returns the number of kernels it launched; group_items sets F's items per tile
void group_shape(int m, int64_t s, DevSeries* S);
int launch_group_prep(const DevSeries& S, double* means, cudaStream_t st);
// and returns the largest number of super-group pairs of one.
size_t group_items(int g, GroupFilter* F);
// Samples group pairs of the join's tiles against the best-so-far into F.probe
// (zeroed).
void launch_group_probe(const DevSeries& S, const DevSearch& Q, const GroupFilter& F,
                        const Tile* tiles, int ntiles, cudaStream_t st);
// F.nsup, F.nlist and F.tcount are zero at launch.  Two kernels.
void launch_group(const DevSeries& S, const DevSearch& Q, const GroupFilter& F, const Tile* tiles,
                  int tile_begin, int tile_end, int num_sms, cudaStream_t st);
// Sets the survivor bits of the sparse tiles (masked cascade).
void launch_group_bits(const DevSeries& S, const DevSearch& Q, const GroupFilter& F,
                       const Tile* tiles, int tile_begin, int num_sms, unsigned int* bits,
                       cudaStream_t st);
// Fast diagonal bound over LB tiles [tile_begin, tile_end) that the group
// filter left dense (every tile when F.tcount is nullptr); survivors leave as
// bits, [tile][word][lag], their tiles are listed in F.dense.  Sparse tiles
// only count their pairs; with clear_sparse their bits are zeroed.
// enumerate_all: no pruning (bounds off).  Persistent: CTAs take tiles from
// the work counter *next (zero at launch).
void launch_lb(const DevSeries& S, const DevSearch& Q, const GroupFilter& F, const Tile* tiles,
               int tile_begin, int tile_end, unsigned int* bits, bool enumerate_all,
               bool clear_sparse, unsigned int* next, int num_sms, cudaStream_t st);
size_t lb_smem_bytes();
// Run filter over the survivor bits of LB tiles [tile_begin, tile_end):
// masked bound, endpoint bound and LB_Keogh for every pair of every run of
// consecutive survivors; pairs that survive go to Q.queue.
void launch_runs(const DevSeries& S, const DevSearch& Q, const Tile* tiles, int tile_begin,
                 int tile_end, const unsigned int* bits, bool masked, bool bounds, int num_sms,
                 cudaStream_t st);
void launch_center(const DevSeries& S, cudaStream_t st);
// 64 features per tile for the learned ordering (features.cu), from the
// profile keys of the series' rows (every row keyed: grid 1; the seed
// profile: grid kSeedGrid); out[64 * t ...] for tile t.
void launch_tile_features(const DevSeries& S, const Tile* tiles, int ntiles,
                          const unsigned long long* keys, int grid, float* out, cudaStream_t st);
// Block-mean lower bound (LB_PAA), then the endpoint bound, over the survivor
// bits of the dense tiles; survivors go to Q.kq.
void launch_paa(const DevSeries& S, const DevSearch& Q, const GroupFilter& F, const Tile* tiles,
                int tile_begin, int tile_end, const unsigned int* bits, int num_sms,
                cudaStream_t st);
// The same over the pairs of the group filter's surviving groups (sparse
// tiles; next: a zeroed work counter).
void launch_paa_groups(const DevSeries& S, const DevSearch& Q, const GroupFilter& F,
                       const Tile* tiles, int tile_begin, int tile_end, unsigned int* next,
                       int num_sms, cudaStream_t st);
// Block length of the block-mean bound for windows of length m.
int paa_block(int m);
// Sliding block means (pq, or pq2 and wrec for windows of at most 1024
// samples), per-block magnitudes (cmax) and per-window error scales (rw);
// after launch_center.  Returns the number of kernels it launched.
int launch_paa_prep(const DevSeries& S, cudaStream_t st);
// LB_Keogh over the candidates the run filter queued in Q.kq; survivors go to
// Q.queue.
void launch_keogh(const DevSeries& S, const DevSearch& Q, int num_sms, cudaStream_t st);
// LB_Petitjean (csrc/petitjean.cu): the join stage filters the DTW queue of a
// chunk in place (next: a zeroed work counter); it runs when one warp's
// shared tables, 2 (m + 2w) doubles, fit kPjMaxSmemBytes.
constexpr size_t kPjMaxSmemBytes = 200 * 1024;
bool petitjean_fits(int m, int w);
void launch_petitjean(const DevSeries& S, const DevSearch& Q, unsigned int* next, int num_sms,
                      cudaStream_t st);
size_t lbp_list_bytes(int m, int w, bool own_env);
void launch_lbp_list(const DevSeries& S, const int2* pairs, int count, bool own_env,
                     double* keogh_mid, double* terms, int num_sms, cudaStream_t st);
// bounds = false: DTW only (the seeds); true: endpoint bound + LB_Keogh first.
// Layouts with up to 8 cells per lane and bounds run in slots (dtw_slots.cuh).
void launch_pairs(const DevSeries& S, const DevSearch& Q, const int2* pairs,
                  const unsigned int* npairs, bool bounds, BandShape band, int num_sms,
                  cudaStream_t st);
void launch_dtw_slots4(int cells, const DevSeries& S, const DevSearch& Q, const int2* pairs,
                       const unsigned int* npairs, int num_sms, int warps, cudaStream_t st);
void launch_dtw_slots8(int cells, const DevSeries& S, const DevSearch& Q, const int2* pairs,
                       const unsigned int* npairs, int num_sms, int warps, cudaStream_t st);
void launch_dtw_slots16(int cells, const DevSeries& S, const DevSearch& Q, const int2* pairs,
                        const unsigned int* npairs, int num_sms, int warps, cudaStream_t st);
void launch_dtw_slots32(int cells, const DevSeries& S, const DevSearch& Q, const int2* pairs,
                        const unsigned int* npairs, int num_sms, int warps, cudaStream_t st);
// Fills the window table if the queue holds more than half as many pairs as
// the series has windows and it is not filled yet.
void launch_window_table(const DevSeries& S, const DevSearch& Q, int num_sms, cudaStream_t st);
// FP64 re-verification of the candidates, then per series the lexicographic
// minimum (d2, i, j): best_d2[series] (FP64 squared distance, +inf if none),
// best_ij[series] = i << 32 | j, best_f32[series] = the search's FP32 d2 (the
// three arrays follow one another).
void launch_verify(const DevSeries& S, const DevSearch& Q, BandShape band, double* out_d2,
                   unsigned long long* best_d2, unsigned long long* best_ij, float* best_f32,
                   cudaStream_t st);
}  // namespace dtwj
struct dtwj_mlp;
namespace dtwj {
// Tile scores for the learned order (mlp.cu): x_dev [count][64] on the
// device, after the work queued on st; y_dev [count].
int mlp_predict_device(dtwj_mlp* net, const float* x_dev, int64_t count, float* y_dev,
                       cudaStream_t st);
int mlp_device(const dtwj_mlp* net);
void launch_pair_dtw(const DevSeries& S, const int2* pairs, int count, bool precise,
                     BandShape band, double* out_d2, cudaStream_t st);

}  // namespace dtwj
