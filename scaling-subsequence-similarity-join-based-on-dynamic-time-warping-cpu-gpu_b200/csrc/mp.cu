// z-normalised Euclidean matrix profile (the reference's mpx_v2) and the
// ED-seeded best-so-far.
//
// mpx_v2 (CPU_version1/mpx_v2.cpp:79-113, GPU_version1/src/mpx_v2.cu:80-115)
// walks every diagonal with the covariance recurrence
//   cov -= dr_bwd * dc_bwd;  cov += dr_fwd * dc_fwd
// on one host thread.  Here one thread owns one lag L and walks a block of
// rows with the equivalent centered FP64 update
//   C(i, j) = C(i-1, j-1) + df[i-1] dg[j-1] + df[j-1] dg[i-1],
// re-anchored exactly at the first row of every tile, and the row minimum of
// ED^2 = 2m - 2 C / (sig_i sig_j) is reduced across the warp in one REDUX.
// A key packs the high 32 bits of ED^2 (sign, exponent, 20 mantissa bits:
// monotone for non-negative doubles; the lowest 3 bits give way to the lag
// inside a thread's minimum) above the partner index, so a 64-bit atomicMin
// keeps the nearest neighbour at that resolution.  That is all the seeds
// need; the matrix profile (dtwj_matrix_profile, k_profile below) decides every
// row at FP64 among the partners whose key is near the row's.
//
// The seeds are the kSeeds smallest row minima, as in
// CPU_version1/new_dtw_motifGUI.cpp:53-74 (min_v_k + exact DTW per seed).
#include "dtwj_dev.cuh"

#include <cfloat>
#include <climits>

namespace dtwj {
namespace {

// Row minima of ED^2 over the upper triangle (partners j >= i + m).  Tile and
// staging as in the diagonal sweep (lb.cu): 128 threads x kLbPerThread lags
// x kLbRows rows, column operands (df[j-1], dg[j-1], 1/sig_j and the flat
// guard 2m | 1e300) staged per kStage rows in shared memory and slid through
// registers.  Per row a thread keeps its best of kLbPerThread lags, the warp
// reduces the high words with one REDUX, and the winner lane folds its key
// into the tile's row minima with a shared 64-bit atomicMin.
constexpr int kStage = kLbPerThread * 32;
constexpr int kCols = kLbLags + kStage;

// High words of ED^2 keys at or above this (ED^2 >= 2^513) come from the
// 1e300 offset of a column past the series or of a flat window, not a pair.
constexpr unsigned int kKeyReal = 0x60000000u;
static_assert(kLbPerThread <= 8, "the lag fits the key's 3 low bits");

struct MpShared {
  double p1[kCols], p2[kCols], is[kCols], c2[kCols];
  double r1[kStage], r2[kStage], ci[kStage];
  unsigned long long rowbest[kStage];  // row minima of the current stage
};

__global__ void __launch_bounds__(kLbThreads, 4) k_mp(DevSeries S, const Tile* tiles,
                                                      unsigned long long* keys,
                                                      unsigned int* tile_best, int tile_base) {
  extern __shared__ __align__(16) unsigned char smraw[];
  MpShared& sh = *reinterpret_cast<MpShared*>(smraw);
  const Tile T = tiles[blockIdx.x];
  const int64_t s = T.send;  // windows of the tile's series end here
  const int m = S.m;
  const int t = threadIdx.x, lane = t & 31;
  const int64_t L0 = T.L0, i0 = T.i0;
  const int64_t Lt = L0 + (int64_t)t * kLbPerThread;

  // exact anchors C(i0, i0 + L) for the thread's lags
  double C[kLbPerThread];
  {
    double mj[kLbPerThread], wa[kLbPerThread];
    const int64_t jb = i0 + Lt;
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) {
      C[l] = 0.0;
      mj[l] = S.mu[jb + l < s ? jb + l : s - 1];
      wa[l] = S.a[jb + l < S.n ? jb + l : S.n - 1];
    }
    const double mi = S.mu[i0];
    for (int k = 0; k < m; ++k) {
      const double ai = S.a[i0 + k] - mi;
#pragma unroll
      for (int l = 0; l < kLbPerThread; ++l) C[l] = fma(ai, wa[l] - mj[l], C[l]);
#pragma unroll
      for (int l = 0; l < kLbPerThread - 1; ++l) wa[l] = wa[l + 1];
      const int64_t x = jb + kLbPerThread + k < S.n ? jb + kLbPerThread + k : S.n - 1;
      wa[kLbPerThread - 1] = S.a[x];
    }
  }
  double w1[kLbPerThread], w2[kLbPerThread], wi[kLbPerThread], wc[kLbPerThread];
  const double two_m = 2.0 * m;
  unsigned int tmin = 0xffffffffu;  // the tile's smallest key (high bits of ED^2)
  for (int st = 0; st < T.rows; st += kStage) {
    const int64_t r0 = i0 + st, c0 = r0 + L0;
    __syncthreads();
    for (int x = t; x < kStage; x += kLbThreads) sh.rowbest[x] = ULLONG_MAX;
    for (int x = t; x < kCols; x += kLbThreads) {
      const int64_t j = c0 + x;
      const bool in = j >= 0 && j < s, up = j >= 1 && j < s;  // update terms exist for j >= 1
      sh.p1[x] = up ? S.dfa[j - 1] : 0.0;
      sh.p2[x] = up ? S.dga[j - 1] : 0.0;
      sh.is[x] = in ? S.isg[j] : 0.0;
      sh.c2[x] = (in && !S.flat[j]) ? two_m : 1e300;
    }
    for (int x = t; x < kStage; x += kLbThreads) {
      const int64_t i = r0 + x;
      const bool in = i >= 0 && i < s, up = i >= 1 && i < s;
      sh.r1[x] = up ? S.dfa[i - 1] : 0.0;
      sh.r2[x] = up ? S.dga[i - 1] : 0.0;
      sh.ci[x] = (in && !S.flat[i]) ? -2.0 * S.isg[i] : 0.0;
    }
    __syncthreads();
    const int cb = t * kLbPerThread;
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) {
      w1[l] = sh.p1[cb + l];
      w2[l] = sh.p2[cb + l];
      wi[l] = sh.is[cb + l];
      wc[l] = sh.c2[cb + l];
    }
    for (int qq = 0; qq < kStage / kLbPerThread; ++qq) {
#pragma unroll
      for (int u = 0; u < kLbPerThread; ++u) {
        const int r = qq * kLbPerThread + u;
        const int64_t i = r0 + r;
        const bool first = (st == 0 && r == 0);
        const double q1 = sh.r1[r], q2 = sh.r2[r], qc = sh.ci[r];
        // rows of the tile with a non-flat window (warp-uniform); a column past
        // the series or flat has weight 0 and offset 1e300, so its key is far
        // above any real one and it never needs a test of its own
        const bool row_ok = (st + r < T.rows) && qc != 0.0;
        unsigned int best = UINT_MAX;
#pragma unroll
        for (int l = 0; l < kLbPerThread; ++l) {
          const int sl = (u + l) % kLbPerThread;
          if (!first) {
            C[l] = fma(q1, w2[sl], C[l]);
            C[l] = fma(w1[sl], q2, C[l]);
          }
          const double e2 = fmax(fma(C[l] * qc, wi[sl], wc[sl]), 0.0);
          const unsigned int hi = (unsigned int)__double2hiint(e2);
          // the high word with its lowest 3 bits replaced by the lag: one
          // minimum keeps the nearest lag (17 mantissa bits of ED^2)
          best = min(best, (hi & ~7u) | (unsigned int)l);
        }
        const int nx = cb + r + kLbPerThread;
        w1[u] = sh.p1[nx];
        w2[u] = sh.p2[nx];
        wi[u] = sh.is[nx];
        wc[u] = sh.c2[nx];
        if (row_ok) {  // flat rows have no neighbour
          const unsigned int wbest = __reduce_min_sync(0xffffffffu, best);
          if (wbest < kKeyReal) {
            const unsigned int ballot = __ballot_sync(0xffffffffu, best == wbest);
            if (lane == __ffs(ballot) - 1) {
              const unsigned long long key =
                  ((unsigned long long)(wbest & ~7u) << 32) |
                  (unsigned long long)(unsigned int)(i + Lt + (wbest & 7u));
              atomicMin(&sh.rowbest[r], key);
            }
          }
        }
      }
    }
    // the stage's row minima into the series' keys (each row once per tile)
    __syncthreads();
    const int nrow = T.rows - st < kStage ? T.rows - st : kStage;
    for (int x = t; x < nrow; x += kLbThreads) {
      const unsigned long long v = sh.rowbest[x];
      if (v != ULLONG_MAX) {
        atomicMin(&keys[r0 + x], v);
        tmin = min(tmin, (unsigned int)(v >> 32));
      }
    }
  }
  if (tile_best) {
    for (int o = 16; o > 0; o >>= 1) tmin = min(tmin, __shfl_xor_sync(0xffffffffu, tmin, o));
    if (lane == 0 && tmin != 0xffffffffu) atomicMin(&tile_best[tile_base + blockIdx.x], tmin);
  }
}

// Row minima for the join's seeds only.  The seeds choose which pairs get an
// exact DTW first; nothing else depends on these keys (the join's starting
// best-so-far comes from those exact DTWs, and the result never depends on
// it), so this pass samples and approximates:
//  - only the rows on a grid of kSeedGrid rows (i - i0 a multiple of
//    kSeedGrid; every tile starts on the grid of its series) get a key.  The
//    covariance recurrence still steps every row, but the ED^2, the minimum
//    and the row reduction run on one row in kSeedGrid.  A seed (i, j) is
//    later widened to its diagonal neighbours (i + d, j + d), |d| <=
//    kSeedGrid / 2, which covers every row of the grid cell;
//  - the pass keeps the tile's exact FP64 anchor and carries the covariance
//    in FP64 from stage to stage, but accumulates the per-row increments of a
//    stage (224 rows) in FP32 on FP32 copies of the update terms.  On random
//    walks that leaves ED^2 within about 1e-4 of the FP64 recurrence; the keys
//    keep 20 mantissa bits.
static_assert(kSeedGrid == kLbPerThread, "grid rows are the first of each unrolled group");
static_assert(kLbRows % kSeedGrid == 0 && kStage % kSeedGrid == 0, "tiles and stages on the grid");

constexpr int kSeedCtasPerSm = 6;  // launch bounds of k_mp_seed

struct MpSeedShared {
  float2 p[kCols];   // (dfa, dga) of column j - 1: one 8-byte read per row and thread
  float is[kCols], c2[kCols];
  float4 r[kStage];  // (dfa, dga of row i - 1, -2 isg of row i, 0): one broadcast read per row
  unsigned long long rowbest[kStage / kSeedGrid];
};

// A block takes `part` stages of a tile (blockIdx.x: tile, blockIdx.y: part of
// it), all 18 when the tiles alone fill the GPU.  Each part starts from its
// own exact anchors, so a tile is cut only as far as that pays (tile_part): a
// series of 20,000 samples has 66 tiles, and one block per tile walks 4,032
// rows one after another on half of the SMs (0.25 ms).
__global__ void __launch_bounds__(kLbThreads, kSeedCtasPerSm) k_mp_seed(DevSeries S,
                                                                      const Tile* tiles, int part,
                                                                      unsigned long long* keys,
                                                                      const unsigned int* walk) {
  extern __shared__ __align__(16) unsigned char smraw[];
  MpSeedShared& sh = *reinterpret_cast<MpSeedShared*>(smraw);
  if (walk && *walk == 0u) return;
  Tile T = tiles[blockIdx.x];
  {
    const int first = (int)blockIdx.y * part * kStage;
    if (first >= T.rows) return;
    T.i0 += first;
    T.rows = T.rows - first < part * kStage ? T.rows - first : part * kStage;
  }
  const int64_t s = T.send;
  const int m = S.m;
  const int t = threadIdx.x, lane = t & 31;
  const int64_t L0 = T.L0, i0 = T.i0;
  const int64_t Lt = L0 + (int64_t)t * kLbPerThread;
  // exact anchors C(i0, i0 + L) = sum_k (a[i0+k] - mu_i) (a[j+k] - mu_j) for the
  // thread's lags (FP64), the samples staged kStage at a time.  The columns
  // are centered on one value c0 near their means when staged, which leaves
  // one multiply-add per lag and sample; sum_k (a[i0+k] - mu_i), zero up to
  // rounding, takes the rest of the centering.
  double C[kLbPerThread];
  {
    double* col = reinterpret_cast<double*>(sh.p);
    double* row = reinterpret_cast<double*>(sh.r);
    static_assert(sizeof sh.p >= kCols * sizeof(double) && sizeof sh.r >= kStage * sizeof(double),
                  "staging fits");
    const double mi = S.mu[i0];
    const double c0 = S.mu[i0 + L0 + kLbLags / 2 < s ? i0 + L0 + kLbLags / 2 : s - 1];
    const int cb = t * kLbPerThread;
    double wa[kLbPerThread], rsum = 0.0;
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) C[l] = 0.0;
    for (int k0 = 0; k0 < m; k0 += kStage) {
      const int cnt = m - k0 < kStage ? m - k0 : kStage;
      __syncthreads();
      for (int x = t; x < kCols; x += kLbThreads) {
        const int64_t q = i0 + L0 + k0 + x;
        col[x] = S.a[q < S.n ? q : S.n - 1] - c0;
      }
      for (int x = t; x < cnt; x += kLbThreads) row[x] = S.a[i0 + k0 + x] - mi;
      __syncthreads();
#pragma unroll
      for (int l = 0; l < kLbPerThread; ++l) wa[l] = col[cb + l];
      int k = 0;
      for (; k + kLbPerThread <= cnt; k += kLbPerThread) {
#pragma unroll
        for (int u = 0; u < kLbPerThread; ++u) {
          const double ai = row[k + u];
          rsum += ai;
#pragma unroll
          for (int l = 0; l < kLbPerThread; ++l) C[l] = fma(ai, wa[(u + l) % kLbPerThread], C[l]);
          wa[u] = col[cb + k + u + kLbPerThread];
        }
      }
      for (; k < cnt; ++k) {
        const double ai = row[k];
        rsum += ai;
#pragma unroll
        for (int l = 0; l < kLbPerThread; ++l) C[l] = fma(ai, col[cb + k + l], C[l]);
      }
    }
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) {
      const int64_t j = i0 + Lt + l < s ? i0 + Lt + l : s - 1;
      C[l] = fma(c0 - S.mu[j], rsum, C[l]);
    }
  }
  float w1[kLbPerThread], w2[kLbPerThread];
  const float two_m = 2.0f * (float)m;
  const unsigned int kReal = __float_as_uint(1e20f);  // above: a guard column, not a pair
  for (int st = 0; st < T.rows; st += kStage) {
    const int64_t r0 = i0 + st, c0 = r0 + L0;
    __syncthreads();
    for (int x = t; x < kStage / kSeedGrid; x += kLbThreads) sh.rowbest[x] = ULLONG_MAX;
    for (int x = t; x < kCols; x += kLbThreads) {
      const int64_t j = c0 + x;
      const bool in = j >= 0 && j < s, up = j >= 1 && j < s;
      sh.p[x] = make_float2(up ? (float)S.dfa[j - 1] : 0.0f, up ? (float)S.dga[j - 1] : 0.0f);
      sh.is[x] = in ? (float)S.isg[j] : 0.0f;
      sh.c2[x] = (in && !S.flat[j]) ? two_m : 1e30f;
    }
    for (int x = t; x < kStage; x += kLbThreads) {
      const int64_t i = r0 + x;
      const bool in = i >= 0 && i < s, up = i >= 1 && i < s;
      sh.r[x] = make_float4(up ? (float)S.dfa[i - 1] : 0.0f, up ? (float)S.dga[i - 1] : 0.0f,
                            (in && !S.flat[i]) ? (float)(-2.0 * S.isg[i]) : 0.0f, 0.0f);
    }
    __syncthreads();
    const int cb = t * kLbPerThread;
    float Cb[kLbPerThread], D[kLbPerThread];
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) {
      const float2 pc = sh.p[cb + l];
      w1[l] = pc.x;
      w2[l] = pc.y;
      Cb[l] = (float)C[l];
      D[l] = 0.0f;
    }
    for (int qq = 0; qq < kStage / kLbPerThread; ++qq) {
#pragma unroll
      for (int u = 0; u < kLbPerThread; ++u) {
        const int r = qq * kLbPerThread + u;
        const bool first = (st == 0 && r == 0);
        const float4 rq = sh.r[r];
        const float q1 = rq.x, q2 = rq.y;
        if (!first) {
#pragma unroll
          for (int l = 0; l < kLbPerThread; ++l) {
            const int sl = (u + l) % kLbPerThread;  // ring slot of lag l at this row
            D[l] = fmaf(q1, w2[sl], D[l]);
            D[l] = fmaf(w1[sl], q2, D[l]);
          }
        }
        // a grid row (u == 0: lag l's column sits in ring slot l and at
        // stage column cb + r + l)
        const float qc = rq.z;
        if (u == 0 && st + r < T.rows && qc != 0.0f) {
          unsigned int best = UINT_MAX;
#pragma unroll
          for (int l = 0; l < kLbPerThread; ++l) {
            const float e2 =
                fmaxf(fmaf((Cb[l] + D[l]) * qc, sh.is[cb + r + l], sh.c2[cb + r + l]), 0.0f);
            best = min(best, (__float_as_uint(e2) & ~7u) | (unsigned int)l);
          }
          const unsigned int wbest = __reduce_min_sync(0xffffffffu, best);
          if (wbest < kReal) {
            const unsigned int ballot = __ballot_sync(0xffffffffu, best == wbest);
            if (lane == __ffs(ballot) - 1) {
              // the float (20 mantissa bits kept) in the FP64 key format
              const unsigned int hi =
                  (unsigned int)__double2hiint((double)__uint_as_float(wbest & ~7u));
              const unsigned long long key =
                  ((unsigned long long)(hi & ~7u) << 32) |
                  (unsigned long long)(unsigned int)(r0 + r + Lt + (wbest & 7u));
              atomicMin(&sh.rowbest[r / kSeedGrid], key);
            }
          }
        }
        const int nx = cb + r + kLbPerThread;
        const float2 pn = sh.p[nx];
        w1[u] = pn.x;
        w2[u] = pn.y;
      }
    }
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) C[l] += (double)D[l];
    __syncthreads();
    const int nrow = T.rows - st < kStage ? T.rows - st : kStage;
    for (int x = t; x * kSeedGrid < nrow; x += kLbThreads) {
      const unsigned long long v = sh.rowbest[x];
      if (v != ULLONG_MAX) atomicMin(&keys[r0 + (int64_t)x * kSeedGrid], v);
    }
  }
}

// Per tile, an upper bound on its smallest squared DTW distance: the ED^2 of
// its closest pair (ED >= DTW), from the truncated key rounded up.
__global__ void k_tile_bound(const unsigned int* tile_best, int ntiles, unsigned int* bsf2) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  const unsigned int hi = tile_best[t];
  if (hi == 0xffffffffu) {
    bsf2[t] = 0x7f800000u;
    return;
  }
  // the key's high word has its 3 low bits cleared: the pair's ED^2 is below
  // the next multiple of 8 units
  const unsigned long long bits = ((unsigned long long)(hi & ~7u) + 8ull) << 32;
  bsf2[t] = __float_as_uint(__double2float_ru(__longlong_as_double((long long)bits)));
}

__global__ void k_fill_u64(unsigned long long* p, int64_t n, unsigned long long v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

// Exact squared distance of candidate pairs (row, partner), one warp per pair.
// pick == false: rowmin[i] = the
// smallest FP64 bits over the row's candidates (non-negative doubles order as
// their bits); pick == true: rowidx[i] = the lowest partner reaching it.
__global__ void k_mp_exact(DevSeries S, const int2* cand, const unsigned int* count,
                           unsigned int cap, bool pick, unsigned long long* rowmin, unsigned long long* rowidx) {
  const int lane = threadIdx.x & 31;
  const unsigned int total = *count < cap ? *count : cap;
  for (unsigned int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < total;
       c += (gridDim.x * blockDim.x) >> 5) {
    const int2 p = cand[c];
    const int64_t i = p.x, j = p.y;
    const double mi = S.mu[i], mj = S.mu[j], si = S.isg[i], sj = S.isg[j];
    double d2 = 0.0;
    for (int q = lane; q < S.m; q += 32) {
      const double d = (S.a[i + q] - mi) * si - (S.a[j + q] - mj) * sj;
      d2 = fma(d, d, d2);
    }
    for (int o = 16; o > 0; o >>= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, o);
    if (lane == 0) {
      const unsigned long long b = (unsigned long long)__double_as_longlong(d2);
      if (!pick) atomicMin(&rowmin[i], b);
      else if (b == rowmin[i]) atomicMin(&rowidx[i], (unsigned long long)j);
    }
  }
}

// mp[i] = sqrt of the row's exact minimum, mpi[i] its lowest partner.
__global__ void k_mp_exact_out(int64_t s, const unsigned long long* rowmin,
                               const unsigned long long* rowidx, double* mp, int64_t* mpi) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= s) return;
  if (rowidx[i] == ULLONG_MAX) {
    mp[i] = __longlong_as_double(0x7ff0000000000000LL);
    mpi[i] = -1;
    return;
  }
  mp[i] = sqrt(__longlong_as_double((long long)rowmin[i]));
  mpi[i] = (int64_t)rowidx[i];
}

// The ED matrix profile (dtwj_matrix_profile): one walk over the upper triangle
// keeps every window's smallest ED^2 as row and as column, a second one lists
// the pairs near either window's smallest.  Walking only rows needed both
// walks on the reversed series as well: 18.3 ms at 100,003 samples and m = 256.
//
// Tile, staging and recurrence are k_mp's.  A column passes through a thread's
// kLbPerThread ring registers from its last lag to its first over as many
// rows, so its minimum costs one integer minimum per pair and one shared
// atomic per row and thread; the keys are the high words of ED^2.
struct ProfShared {
  double p1[kCols], p2[kCols], is[kCols], c2[kCols];
  double r1[kStage], r2[kStage], ci[kStage];
  unsigned int row[kStage], col[kCols];  // minima of the stage, or limits (COLLECT)
};
constexpr int kProfCtasPerSm = 4;  // launch bounds of k_profile
struct ProfOut {
  unsigned int* best;  // per window: smallest high word (also what COLLECT reads)
  int2* up;            // (row, later partner) and (row, earlier partner) near the row's best
  int2* lo;
  unsigned int* count;  // [2]
  unsigned int cap;
};

// The largest high word of ED^2 at which a pair is listed for a window whose
// smallest is `best` (UINT_MAX: none).  Two words are within two units of each
// other when their ED^2 are within 2^-19; ten units leave room for the
// recurrence's relative rounding.  Near zero, where ED^2 is a difference of
// equal terms, its absolute rounding counts: each of up to kLbRows rows rounds
// twice by 2^-53 of a covariance of at most m sig_i sig_j, the anchor's m terms
// once, so two pairs of equal distance are within 2 m (2^-39 + m 2^-52).  The
// row and the column minimum of a window come from different places of their
// tiles and round differently, also for bitwise equal partners.
__device__ __forceinline__ unsigned int near_limit(unsigned int best, int m) {
  if (best == UINT_MAX) return 0u;
  const double e2 = __hiloint2double((int)best, 0) + m * (0x1p-38 + m * 0x1p-51);
  return (unsigned int)__double2hiint(e2) + 10u;
}

template <bool COLLECT>
__global__ void __launch_bounds__(kLbThreads, kProfCtasPerSm) k_profile(DevSeries S,
                                                                      const Tile* tiles, int part,
                                                                      ProfOut out) {
  extern __shared__ __align__(16) unsigned char smraw[];
  ProfShared& sh = *reinterpret_cast<ProfShared*>(smraw);
  Tile T = tiles[blockIdx.x];
  {  // this block's stages of the tile
    const int first = (int)blockIdx.y * part * kStage;
    if (first >= T.rows) return;
    T.i0 += first;
    T.rows = T.rows - first < part * kStage ? T.rows - first : part * kStage;
  }
  const int64_t s = T.send;
  const int m = S.m;
  const int t = threadIdx.x, lane = t & 31;
  const int64_t L0 = T.L0, i0 = T.i0;
  const int64_t Lt = L0 + (int64_t)t * kLbPerThread;
  const int cb = t * kLbPerThread;
  // exact anchors C(i0, i0 + L) for the thread's lags, the samples staged
  // kStage at a time
  double C[kLbPerThread];
  {
    double mj[kLbPerThread];
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) {
      C[l] = 0.0;
      mj[l] = S.mu[i0 + Lt + l < s ? i0 + Lt + l : s - 1];
    }
    const double mi = S.mu[i0];
    for (int k0 = 0; k0 < m; k0 += kStage) {
      const int cnt = m - k0 < kStage ? m - k0 : kStage;
      __syncthreads();
      for (int x = t; x < kCols; x += kLbThreads) {
        const int64_t q = i0 + L0 + k0 + x;
        sh.p1[x] = S.a[q < S.n ? q : S.n - 1];
      }
      for (int x = t; x < cnt; x += kLbThreads) sh.r1[x] = S.a[i0 + k0 + x] - mi;
      __syncthreads();
#pragma unroll 2
      for (int k = 0; k < cnt; ++k) {
        const double ai = sh.r1[k];
#pragma unroll
        for (int l = 0; l < kLbPerThread; ++l) C[l] = fma(ai, sh.p1[cb + k + l] - mj[l], C[l]);
      }
    }
  }
  double w1[kLbPerThread], w2[kLbPerThread], wi[kLbPerThread], wc[kLbPerThread];
  unsigned int wm[kLbPerThread];  // the ring columns' minima, or limits
  const double two_m = 2.0 * m;
  for (int st = 0; st < T.rows; st += kStage) {
    const int64_t r0 = i0 + st, c0 = r0 + L0;
    __syncthreads();
    for (int x = t; x < kCols; x += kLbThreads) {
      const int64_t j = c0 + x;
      const bool in = j < s, up = j >= 1 && in;  // update terms exist for j >= 1
      sh.p1[x] = up ? S.dfa[j - 1] : 0.0;
      sh.p2[x] = up ? S.dga[j - 1] : 0.0;
      sh.is[x] = in ? S.isg[j] : 0.0;
      // a column past the series or flat: no weight, an offset no pair reaches
      sh.c2[x] = (in && !S.flat[j]) ? two_m : 1e300;
      sh.col[x] = COLLECT ? near_limit(in ? out.best[j] : UINT_MAX, m) : UINT_MAX;
    }
    for (int x = t; x < kStage; x += kLbThreads) {
      const int64_t i = r0 + x;
      const bool in = i < s, up = i >= 1 && in;
      sh.r1[x] = up ? S.dfa[i - 1] : 0.0;
      sh.r2[x] = up ? S.dga[i - 1] : 0.0;
      sh.ci[x] = (in && !S.flat[i]) ? -2.0 * S.isg[i] : 0.0;
      sh.row[x] = COLLECT ? near_limit(in ? out.best[i] : UINT_MAX, m) : UINT_MAX;
    }
    __syncthreads();
#pragma unroll
    for (int l = 0; l < kLbPerThread; ++l) {
      w1[l] = sh.p1[cb + l];
      w2[l] = sh.p2[cb + l];
      wi[l] = sh.is[cb + l];
      wc[l] = sh.c2[cb + l];
      wm[l] = COLLECT ? sh.col[cb + l] : UINT_MAX;
    }
    for (int qq = 0; qq < kStage / kLbPerThread; ++qq) {
#pragma unroll
      for (int u = 0; u < kLbPerThread; ++u) {
        const int r = qq * kLbPerThread + u;
        const int64_t i = r0 + r;
        const double q1 = sh.r1[r], q2 = sh.r2[r], qc = sh.ci[r];
        // rows of the tile with a non-flat window (warp-uniform)
        const bool row_ok = (st + r < T.rows) && qc != 0.0;
        if (st > 0 || r > 0) {
#pragma unroll
          for (int l = 0; l < kLbPerThread; ++l) {
            const int sl = (u + l) % kLbPerThread;
            C[l] = fma(q1, w2[sl], C[l]);
            C[l] = fma(w1[sl], q2, C[l]);
          }
        }
        if (row_ok) {
          const unsigned int lim = COLLECT ? sh.row[r] : 0u;
          unsigned int best = UINT_MAX, hs[kLbPerThread];
          bool hit = false;  // one branch per row: candidates are rare
#pragma unroll
          for (int l = 0; l < kLbPerThread; ++l) {
            const int sl = (u + l) % kLbPerThread;
            // below zero only by rounding
            const int h = __double2hiint(fma(C[l] * qc, wi[sl], wc[sl]));
            const unsigned int hi = (unsigned int)max(h, 0);
            if (COLLECT) {
              hs[l] = hi;
              hit = hit || hi <= max(lim, wm[sl]);
            } else {
              best = min(best, hi);
              wm[sl] = min(wm[sl], hi);
            }
          }
          if (COLLECT && hit) {
#pragma unroll
            for (int l = 0; l < kLbPerThread; ++l) {
              const int j = (int)(i + Lt + l);
              if (hs[l] <= lim) {
                const unsigned int slot = atomicAdd(out.count, 1u);
                if (slot < out.cap) out.up[slot] = make_int2((int)i, j);
              }
              if (hs[l] <= wm[(u + l) % kLbPerThread]) {
                const unsigned int slot = atomicAdd(out.count + 1, 1u);
                if (slot < out.cap) out.lo[slot] = make_int2(j, (int)i);
              }
            }
          }
          if (!COLLECT) {
            best = __reduce_min_sync(0xffffffffu, best);
            if (lane == 0) atomicMin(&sh.row[r], best);
          }
        }
        // lag 0's column leaves the thread (a stage's last ones below)
        const int nx = cb + r + kLbPerThread;
        if (!COLLECT) atomicMin(&sh.col[nx - kLbPerThread], wm[u]);
        w1[u] = sh.p1[nx];
        w2[u] = sh.p2[nx];
        wi[u] = sh.is[nx];
        wc[u] = sh.c2[nx];
        wm[u] = COLLECT ? sh.col[nx] : UINT_MAX;
      }
    }
    if (!COLLECT) {
      // ring slot l holds column kStage + l (kStage rows are whole turns)
#pragma unroll
      for (int l = 0; l < kLbPerThread; ++l) atomicMin(&sh.col[cb + kStage + l], wm[l]);
      __syncthreads();
      for (int x = t; x < kStage; x += kLbThreads)
        if (sh.row[x] < kKeyReal) atomicMin(&out.best[r0 + x], sh.row[x]);
      for (int x = t; x < kCols; x += kLbThreads)
        if (sh.col[x] < kKeyReal) atomicMin(&out.best[c0 + x], sh.col[x]);
    }
  }
}

constexpr int kSelThreads = 1024;

// kSeeds smallest row minima of a series (by ED^2 key, then row index), among
// the rows of the seed grid: the keys' high words are narrowed to the kSeeds-th
// smallest by four rounds of an 8-bit radix select in shared memory, then the
// keys below it are taken, and of those equal to it the lowest rows.  Writes
// each seed pair with its diagonal neighbours (kSeedSpread slots per seed,
// (-1, -1) where a neighbour leaves the series) and the seed count.
__global__ void __launch_bounds__(kSelThreads) k_seed_select(DevSeries S,
                                                              const unsigned long long* keys,
                                                              int2* seeds, unsigned int* nseeds) {
  // block b selects the seeds of series b (windows [wb, we))
  const int b = blockIdx.x, t = threadIdx.x, lane = t & 31;
  const int64_t wb = S.sbeg ? S.sbeg[b] : 0;
  const int64_t we = S.sbeg ? S.sbeg[b + 1] - S.m + 1 : S.s;
  const int64_t rows = (we - wb + kSeedGrid - 1) / kSeedGrid;  // of the grid
  seeds += (size_t)b * kSeedSlots;
  for (int x = t; x < kSeedSlots; x += kSelThreads) seeds[x] = make_int2(-1, -1);
  __shared__ unsigned int hist[256];
  __shared__ unsigned int bin, below, taken, equal_base, wcount[kSelThreads / 32];
  // prefix = the digits of the kSeeds-th smallest high word found so far;
  // need = how many of the keys with that prefix are still to take
  unsigned int prefix = 0, need = kSeeds;
  for (int shift = 24; shift >= 0; shift -= 8) {
    if (t < 256) hist[t] = 0;
    __syncthreads();
    for (int64_t r = t; r < rows; r += 4 * kSelThreads) {
      unsigned int h[4];  // four loads in flight
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t ru = r + u * kSelThreads;
        h[u] = ru < rows ? (unsigned int)(keys[wb + ru * kSeedGrid] >> 32) : 0xffffffffu;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (h[u] == 0xffffffffu) continue;  // no neighbour
        if (shift == 24 || (h[u] >> (shift + 8)) == prefix)
          atomicAdd(&hist[(h[u] >> shift) & 255u], 1u);
      }
    }
    __syncthreads();
    if (t < 32) {
      // lane l sums bins 8 l .. 8 l + 7, a scan finds the lane and bin that
      // reach `need` (none: fewer keys than that, the last bin stands)
      unsigned int c[8], sum = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) sum += (c[q] = hist[8 * t + q]);
      unsigned int inc = sum;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (t >= o) inc += v;
      }
      const unsigned int reach = __ballot_sync(0xffffffffu, inc >= need);
      const int who = reach ? __ffs(reach) - 1 : 31;
      if (t == who) {
        unsigned int acc = inc - sum;
        int q = 0;
        while (q < 7 && acc + c[q] < need) acc += c[q++];
        bin = 8u * (unsigned int)t + (unsigned int)q;
        below = acc;
      }
    }
    __syncthreads();
    prefix = (prefix << 8) | bin;
    need = need > below ? need - below : 0u;
    __syncthreads();
  }
  if (t == 0) taken = 0, equal_base = 0;
  __syncthreads();
  // every key below the threshold, and the first `need` rows equal to it
  unsigned long long ahead = t < rows ? keys[wb + (int64_t)t * kSeedGrid] : ULLONG_MAX;
  for (int64_t r0 = 0; r0 < rows; r0 += kSelThreads) {
    const int64_t r = r0 + t, rn = r + kSelThreads;
    const unsigned long long k = ahead;
    ahead = rn < rows ? keys[wb + rn * kSeedGrid] : ULLONG_MAX;
    const unsigned int h = (unsigned int)(k >> 32);
    const bool eq = h == prefix && h != 0xffffffffu;
    bool take = h < prefix;
    if (__syncthreads_or(eq)) {
      const unsigned int eb = __ballot_sync(0xffffffffu, eq);
      if (lane == 0) wcount[t >> 5] = __popc(eb);
      __syncthreads();
      unsigned int rank = equal_base + __popc(eb & ((1u << lane) - 1u));
      for (int w = 0; w < (t >> 5); ++w) rank += wcount[w];
      take = take || (eq && rank < need);
      __syncthreads();
      if (t == 0)
        for (int w = 0; w < kSelThreads / 32; ++w) equal_base += wcount[w];
    }
    if (take) {
      const unsigned int slot = atomicAdd(&taken, 1u);
      const int i = (int)(wb + r * kSeedGrid), pj = (int)(k & 0xffffffffu);
      const int lo = i < pj ? i : pj, hi = i < pj ? pj : i;
      // the pair and its diagonal neighbours that lie in the series
      for (int d = 0; d < kSeedSpread; ++d) {
        const int off = d - kSeedSpread / 2;
        // (a flat window has no z-normalisation: no pair of the join holds one)
        const bool ok = lo + off >= wb && hi + off < we && !S.flat[lo + off] && !S.flat[hi + off];
        seeds[slot * kSeedSpread + d] = ok ? make_int2(lo + off, hi + off) : make_int2(-1, -1);
      }
    }
  }
  __syncthreads();
  if (t == 0) nseeds[b] = taken;
}

}  // namespace

namespace {
constexpr int kStages = kLbRows / kStage;
// Stages of a tile per block.  A block's time alone is its anchors (m rows) and
// `part` stages of kStage rows, a row costing kRowCost anchor rows: 12 us per
// stage and 8 us of anchors at m = 256, nearly all of it latency.  Blocks that
// share an SM hide each other's, so r blocks per SM take 0.75 + r / 3 times
// that (fits r = 1 .. 29 within 15 % for k_mp_seed, and k_profile's best parts
// within 9 %).  Walks of k_mp_seed, against a rule that counted an SM as full
// with four warps: 20,000 samples at m = 256 (66 tiles) 6 -> 2 stages, 110 ->
// 70 us; 30,000 at m = 64 9 -> 1, 153 -> 107 us; 40,000 at m = 400 18 -> 3,
// 298 -> 205 us.  dtwj_matrix_profile of 50,000 at m = 512 18 -> 6, 3.79 ->
// 3.35 ms.
constexpr double kRowCost = 1.75;
int tile_part(int64_t ntiles, int m, int num_sms) {
  int part = kStages;
  double best = 0.0;
  for (int p = kStages; p >= 1; --p) {
    const double r = (double)(ntiles * ((kStages + p - 1) / p)) / num_sms;
    const double load = 0.75 + r / 3.0;
    const double cost = (load > 1.0 ? load : 1.0) * ((double)m + kRowCost * kStage * p);
    if (p == kStages || cost < best) best = cost, part = p;
  }
  return part;
}
}  // namespace

void launch_tile_bound(const unsigned int* tile_best, int ntiles, unsigned int* bsf2,
                       cudaStream_t st) {
  if (ntiles > 0) k_tile_bound<<<(ntiles + 255) / 256, 256, 0, st>>>(tile_best, ntiles, bsf2);
}

void launch_mp(const DevSeries& S, const Tile* tiles, int ntiles, unsigned long long* keys,
               cudaStream_t st, unsigned int* tile_best) {
  k_fill_u64<<<1024, 256, 0, st>>>(keys, S.s, ULLONG_MAX);
  if (ntiles <= 0) return;
  cudaFuncSetAttribute(k_mp, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(MpShared));
  const int slab = 1 << 20;
  for (int b = 0; b < ntiles; b += slab) {
    const int cnt = ntiles - b < slab ? ntiles - b : slab;
    k_mp<<<cnt, kLbThreads, sizeof(MpShared), st>>>(S, tiles + b, keys, tile_best, b);
  }
}

void launch_mp_seed(const DevSeries& S, const Tile* tiles, int ntiles, unsigned long long* keys,
                    const unsigned int* walk, int num_sms, cudaStream_t st) {
  if (!walk) cudaMemsetAsync(keys, 0xff, (size_t)S.s * 8, st);
  if (ntiles <= 0) return;
  cudaFuncSetAttribute(k_mp_seed, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(MpSeedShared));
  const int part = tile_part(ntiles, S.m, num_sms);
  const int parts = (kStages + part - 1) / part;
  const int slab = 1 << 20;
  for (int b = 0; b < ntiles; b += slab) {
    const int cnt = ntiles - b < slab ? ntiles - b : slab;
    k_mp_seed<<<dim3((unsigned)cnt, (unsigned)parts), kLbThreads, sizeof(MpSeedShared), st>>>(
        S, tiles + b, part, keys, walk);
  }
}

void launch_profile(const DevSeries& S, const Tile* tiles, int ntiles, bool collect,
                    unsigned int* best, int2* up, int2* lo, unsigned int* count, unsigned int cap,
                    int num_sms, cudaStream_t st) {
  auto kern = collect ? k_profile<true> : k_profile<false>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ProfShared));
  const ProfOut out = {best, up, lo, count, cap};
  const int part = tile_part(ntiles, S.m, num_sms);
  const unsigned parts = (unsigned)((kStages + part - 1) / part);
  const int slab = 1 << 20;
  for (int b = 0; b < ntiles; b += slab) {
    const int cnt = ntiles - b < slab ? ntiles - b : slab;
    kern<<<dim3((unsigned)cnt, parts), kLbThreads, sizeof(ProfShared), st>>>(S, tiles + b, part,
                                                                             out);
  }
}

void launch_mp_exact(const DevSeries& S, const int2* cand, const unsigned int* count,
                     unsigned int cap, bool pick, unsigned long long* rowmin,
                     unsigned long long* rowidx, cudaStream_t st) {
  k_mp_exact<<<148 * 8, 256, 0, st>>>(S, cand, count, cap, pick, rowmin, rowidx);
}

void launch_mp_exact_out(int64_t s, const unsigned long long* rowmin,
                         const unsigned long long* rowidx, double* mp, int64_t* mpi,
                         cudaStream_t st) {
  k_mp_exact_out<<<(unsigned)((s + 255) / 256), 256, 0, st>>>(s, rowmin, rowidx, mp, mpi);
}

void launch_seed_select(const DevSeries& S, const unsigned long long* keys, int2* seeds,
                        unsigned int* nseeds, cudaStream_t st) {
  k_seed_select<<<S.nseries, kSelThreads, 0, st>>>(S, keys, seeds, nseeds);
}

}  // namespace dtwj
