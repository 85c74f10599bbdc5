// Block-mean bound for groups of windows: the first filter of the sweep.
//
// The block-mean bound of a pair of windows (paa.cu) is
//   LB_PAA = B sum_k max(q_k - U_k, L_k - q_k, 0)^2  <=  LB_Keogh  <=  DTW^2,
// with q_k the mean of the query window over its k-th block of B samples and
// U_k, L_k the means of the other window's envelope, all z-normalised.
// Consecutive windows have nearly the same block means, so a group of g of
// them is described by four numbers per block: the smallest and largest q_k,
// the largest U_k and the smallest L_k over the group.  For two groups I, J
//   max(qmin_I - Umax_J, Lmin_J - qmax_I, 0) <= max(q_k - U_k, L_k - q_k, 0)
// for every window pair in I x J, so one evaluation (in both directions)
// bounds g^2 pairs.  On random walks the group bound settles nearly all of
// them: 99.9 % at m = 1024, w = 52, g = 8 and 98.2 % at m = 512, w = 52 (CPU
// measurement over sampled group pairs), in two to four blocks on average.
// Two levels: super-groups of kGrpFan groups first (g = 32 leaves 0.9 % and
// 13 % of those pairs), then the group pairs of the survivors.
//
// The diagonal bound (lb.cu) judges one pair per 6 FP64 operations and leaves
// 5 % of them; here 1024 pairs (then 64) cost 8 FP32 instructions per block.  Only tiles
// whose groups mostly survive (kDenseNum / kDenseDen) go through the diagonal
// bound; in the others the pairs of the surviving groups go straight to the
// block-mean bound of single pairs (k_paa_groups).
//
// Records are FP32, rounded outward from FP64 (qmin, Lmin down, qmax, Umax
// up).  The FP64 means are of samples relative to the segment's first one, so
// they round by 2^-53 of the window's own range, whatever its level (of samples
// as they are, they were off by a thousandth of a deviation of 1e-12 of the
// level, and pruned pairs).  What is left is the evaluation: each term is off
// by 2^-24 relative and the sum by (terms + 2) 2^-24 < 3e-6, inside the 1/512
// the threshold keeps above the best-so-far.
#include "dtwj_dev.cuh"

#include <cfloat>

namespace dtwj {
namespace {

constexpr int kThreads = 256;
// Record of a window group that must never survive (padding, all windows
// flat): every difference is about 1e15, its square 1e30.
constexpr float kFar = 1e15f;

struct SegOrder {
  unsigned char seg[kGrpSlots];  // segment of slot x; 255: a padding slot
};

// Means of the series and its envelope over [p, p + B) less sample p, FP64: [3][n].
__global__ void k_seg_means(DevSeries S, int B, double* gm) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p + B > S.n) return;
  const double c = S.a[p];
  double sa = 0.0, su = 0.0, sl = 0.0;
  for (int k = 0; k < B; ++k) {
    sa += S.a[p + k] - c;
    su += S.U[p + k] - c;
    sl += S.L[p + k] - c;
  }
  const double ib = 1.0 / (double)B;
  gm[p] = sa * ib;
  gm[S.n + p] = su * ib;
  gm[2 * S.n + p] = sl * ib;
}

// Group records, one thread per (group, slot); consecutive threads take
// consecutive groups, so a warp reads 32 g consecutive means.
__global__ void k_group_rec(DevSeries S, const double* gm, SegOrder ord) {
  const int64_t G = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (G >= S.grp_n) return;
  const int slot = blockIdx.y;
  float4 rec = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int seg = ord.seg[slot];
  if (seg != 255) {
    double qlo = 1e300, qhi = -1e300, up = -1e300, lo = 1e300;
    const int64_t i0 = G * S.grp_g;
    for (int e = 0; e < S.grp_g; ++e) {
      const int64_t i = i0 + e;
      if (i >= S.s || S.flat[i]) continue;
      const double mu = S.mu[i], is = S.isg[i];
      const int64_t p = i + (int64_t)seg * S.grp_b;
      const double c = S.a[p] - mu, q = (gm[p] + c) * is;
      qlo = fmin(qlo, q);
      qhi = fmax(qhi, q);
      up = fmax(up, (gm[S.n + p] + c) * is);
      lo = fmin(lo, (gm[2 * S.n + p] + c) * is);
    }
    if (qlo <= qhi)
      rec = make_float4(__double2float_rd(qlo), __double2float_ru(qhi), __double2float_ru(up),
                        __double2float_rd(lo));
    else
      rec = make_float4(kFar, -kFar, -kFar, kFar);
  }
  S.grp[(int64_t)slot * S.grp_n + G] = rec;
}

// One segment of a group pair: both directions of the block-mean bound, or
// (ED) the bound on the z-normalised Euclidean distance of the group's pairs,
// whose envelopes are the windows themselves.
template <bool ED>
__device__ __forceinline__ void group_terms(const float4 i, const float4 j, float& a1, float& a2) {
  if (ED) {
    const float d = max3f(i.x - j.y, j.x - i.y, 0.0f);
    a1 = fmaf(d, d, a1);
    return;
  }
  const float d1 = max3f(i.x - j.z, j.w - i.y, 0.0f);
  a1 = fmaf(d1, d1, a1);
  const float d2 = max3f(j.x - i.z, i.w - j.y, 0.0f);
  a2 = fmaf(d2, d2, a2);
}

// Appends the entries of the lanes with `on` to the list (every lane calls).
__device__ __forceinline__ unsigned int append_slot(bool on, int lane, unsigned int* count) {
  const unsigned int b = __ballot_sync(0xffffffffu, on);
  unsigned int base = 0;
  if (lane == 0 && b) base = atomicAdd(count, (unsigned int)__popc(b));
  return __shfl_sync(0xffffffffu, base, 0) + __popc(b & ((1u << lane) - 1u));
}

// First level, super-groups of kGrpFan g windows: one warp takes kSupRows
// consecutive row groups against kSupCols column groups, which hold the
// groups with lags of the tile; a lane takes 2 rows and every eighth column.
// The slots are in an order that spreads the first ones over the window; the
// warp votes every four.
//
// A record is 16 bytes per lane, and a load returns 128 bytes per clock to an
// SM's registers whatever the lanes share, so a lane's 2 x 5 group pairs take
// 28 clocks of loads for 20 of arithmetic, where one row per load and lane
// took 32 for 8: 139 -> 80 us per chunk of 1776 tiles at m = 1024.
constexpr int kSupRows = 8;
constexpr int kSupLaneCols = 5;
constexpr int kSupCols = 8 * kSupLaneCols;
template <bool ED>
__global__ void __launch_bounds__(kThreads) k_group_super(DevSeries S, DevSearch Q, GroupFilter F,
                                                          const Tile* tiles, unsigned int total) {
  const int lane = threadIdx.x & 31;
  const unsigned int item = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (item >= total) return;
  const unsigned int walk = ED ? *F.walk : 0u;
  // (looked at behind the first records: a wait for it here costs 3 % of the pass)
  const bool skip = group_off(F, ED, seed_share(S.grp_g)) | (walk != 0u);
  const unsigned int per = (unsigned int)(F.nib * F.nw);
  const unsigned int tk = item / per, rem = item - tk * per;
  const Tile T = tiles[tk];
  const int g = kGrpFan * S.grp_g;
  const int row0 = (int)(rem / (unsigned)F.nw) * kSupRows + 2 * (lane >> 3);  // of this lane
  const int Ia = T.i0 / g, last_row = T.i0 + T.rows - 1;
  if ((Ia + (int)(rem / (unsigned)F.nw) * kSupRows) * (int64_t)g > last_row) return;
  const int I = Ia + row0;
  const int J = I - 2 * (lane >> 3) + T.L0 / g + (int)(rem % (unsigned)F.nw) * kSupCols + (lane & 7);
  // the pairs that hold pairs of the tile (group_pair_in_tile, the rows' part once)
  unsigned int alive = 0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int ia = (I + r) * g;
    const int lo = ia > T.i0 ? ia : T.i0, hi = ia + g - 1 < last_row ? ia + g - 1 : last_row;
#pragma unroll
    for (int q = 0; q < kSupLaneCols; ++q) {
      const int ja = (J + 8 * q) * g;
      if (lo <= hi && ja < T.send && ja + g - 1 - lo >= T.L0 && ja - hi < T.L0 + kLbLags)
        alive |= 1u << (r * kSupLaneCols + q);
    }
  }
  if (!__any_sync(0xffffffffu, alive != 0u)) return;
  const float thr = ED ? *F.cut : prune_threshold_now(Q.bsf2 + T.series, S.m);
  const float fb = (float)S.grp_b;
  const int64_t n = S.sup_n;
  // addresses past the last record repeat it (those group pairs are not
  // alive); the records run past the last row group by kSupRows and more
  const float4* pi = S.sup + I;
  const float4* pj[kSupLaneCols];
  float a1[2][kSupLaneCols], a2[2][kSupLaneCols];
#pragma unroll
  for (int q = 0; q < kSupLaneCols; ++q) {
    pj[q] = S.sup + (J + 8 * q < n ? J + 8 * q : n - 1);
    a1[0][q] = a1[1][q] = a2[0][q] = a2[1][q] = 0.0f;
  }
#pragma unroll 1
  for (int s0 = 0; s0 < S.grp_d; s0 += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 i0 = pi[0], i1 = pi[1];
      pi += n;
#pragma unroll
      for (int q = 0; q < kSupLaneCols; ++q) {
        const float4 j = *pj[q];
        pj[q] += n;
        group_terms<ED>(i0, j, a1[0][q], a2[0][q]);
        group_terms<ED>(i1, j, a1[1][q], a2[1][q]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int q = 0; q < kSupLaneCols; ++q)
        if (fb * fmaxf(a1[r][q], a2[r][q]) > thr) alive &= ~(1u << (r * kSupLaneCols + q));
    if (skip || !__any_sync(0xffffffffu, alive != 0u)) return;
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int q = 0; q < kSupLaneCols; ++q) {
      const bool on = (alive >> (r * kSupLaneCols + q)) & 1u;
      const unsigned int slot = append_slot(on, lane, F.nsup);
      if (on && slot < F.sup_cap)
        F.sup[slot] = group_code(tk, row0 + r, J + 8 * q - (I + r) - T.L0 / g);
    }
}

// Second level: four lanes per surviving super-group pair, each 2 x 2 of its
// kGrpFan x kGrpFan group pairs (four records for four pairs; one pair per
// lane took two for one).
template <bool ED>
__global__ void __launch_bounds__(kThreads) k_group(DevSeries S, DevSearch Q, GroupFilter F,
                                                    const Tile* tiles) {
  static_assert(kGrpFan == 4, "16 group pairs, four lanes");
  const int lane = threadIdx.x & 31, ha = (lane >> 1) & 1, hb = lane & 1;
  const unsigned int total = *F.nsup < F.sup_cap ? *F.nsup : F.sup_cap;
  const int g = S.grp_g, G = kGrpFan * g;
  const float fb = (float)S.grp_b;
  const int64_t n = S.grp_n;
  for (unsigned int e0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 8; e0 < total;
       e0 += ((gridDim.x * blockDim.x) >> 5) * 8) {
    const unsigned int e = e0 + (lane >> 2);
    const unsigned int code = F.sup[e < total ? e : total - 1];
    const unsigned int tk = group_code_tile(code);
    const Tile T = tiles[tk];
    const GroupPair p = group_code_pair(code, T, G);
    const int I = p.I * kGrpFan + 2 * ha, J = p.J * kGrpFan + 2 * hb;
    unsigned int alive = 0;  // bit 2 r + q: groups I + r, J + q
    if (e < total) {
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (group_pair_in_tile(T, g, I + (x >> 1), J + (x & 1))) alive |= 1u << x;
    }
    const float thr = ED ? *F.cut : prune_threshold_now(Q.bsf2 + T.series, S.m);
    // the records run past the last group by more than a super-group
    const float4* pi = S.grp + (I < n - 1 ? I : n - 2);
    const float4* pj = S.grp + (J < n - 1 ? J : n - 2);
    float a1[4], a2[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) a1[x] = a2[x] = 0.0f;
#pragma unroll 1
    for (int s0 = 0; s0 < S.grp_d && __any_sync(0xffffffffu, alive != 0u); s0 += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 i0 = pi[0], i1 = pi[1], j0 = pj[0], j1 = pj[1];
        pi += n;
        pj += n;
        group_terms<ED>(i0, j0, a1[0], a2[0]);
        group_terms<ED>(i0, j1, a1[1], a2[1]);
        group_terms<ED>(i1, j0, a1[2], a2[2]);
        group_terms<ED>(i1, j1, a1[3], a2[3]);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (fb * fmaxf(a1[x], a2[x]) > thr) alive &= ~(1u << x);
    }
    // the 16 pairs of the super-group pair: row 2 ha + r, column 2 hb + q
    unsigned int mask = ((alive & 3u) << (8 * ha + 2 * hb)) |
                        ((alive >> 2 & 3u) << (8 * ha + 4 + 2 * hb));
    mask |= __shfl_xor_sync(0xffffffffu, mask, 1);
    mask |= __shfl_xor_sync(0xffffffffu, mask, 2);
    const bool on = (lane & 3) == 0 && mask != 0u;
    const unsigned int slot = append_slot(on, lane, F.nlist);
    if (on && slot < F.list_cap) F.list[slot] = make_uint2(code, mask);
    if (on) atomicAdd(ED ? F.tcount : F.tcount + tk, (unsigned int)__popc(mask));
  }
}

// Whether the bound settles anything.  On white noise it settles nothing, its two
// levels are extra work (70,000 samples of noise, m = 512, w = 0: 7.6 ms with
// them, 5.1 without), and the seeds' lists of group pairs overflow (100,003
// samples, m = 256: 8.7 ms for the seeds, walking the diagonals takes 1.1).  A
// sample of the pairs of the join's tiles, one per warp (a lane per segment) and
// spread over the tiles, decides first (group_off).  Pairs without a threshold
// yet don't count.
constexpr int kProbeSamples = 1024;
template <bool ED>
__global__ void __launch_bounds__(kThreads) k_group_probe(DevSeries S, DevSearch Q, GroupFilter F,
                                                          const Tile* tiles, int ntiles) {
  static_assert(kGrpSlots == 32, "a lane per slot");
  const int lane = threadIdx.x & 31;
  const unsigned int x = (blockIdx.x * kThreads + threadIdx.x) / 32;
  const Tile T = tiles[(unsigned long long)x * ntiles / kProbeSamples];
  unsigned int h = x * 0x9e3779b1u;  // a row and a lag of the tile
  h = (h ^ (h >> 15)) * 0x85ebca77u;
  h ^= h >> 13;
  const int row = (int)(h % (unsigned)T.rows), lag = (int)(h / (unsigned)T.rows % kLbLags);
  const int64_t i = T.i0 + row, j = i + T.L0 + lag;
  const float thr = ED ? *F.cut : prune_threshold_now(Q.bsf2 + T.series, S.m);
  const bool counts = j < T.send && thr < __int_as_float(0x7f800000);
  float a1 = 0.0f, a2 = 0.0f;
  if (counts && lane < S.grp_d)
    group_terms<ED>(S.grp[lane * S.grp_n + i / S.grp_g], S.grp[lane * S.grp_n + j / S.grp_g], a1,
                    a2);
  for (int o = 16; o > 0; o >>= 1) {
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
    a2 += __shfl_xor_sync(0xffffffffu, a2, o);
  }
  const bool alive = !((float)S.grp_b * fmaxf(a1, a2) > thr);
  const int all = __syncthreads_count(lane == 0 && counts);
  const int left = __syncthreads_count(lane == 0 && counts && alive);
  if (threadIdx.x == 0) {
    if (all) atomicAdd(&F.probe[0], (unsigned int)all);
    if (left) atomicAdd(&F.probe[1], (unsigned int)left);
  }
}

// The masked cascade reads survivor bits: the pairs of the surviving groups
// of the sparse tiles, set in the bits the diagonal sweep cleared for them.
__global__ void k_group_bits(DevSeries S, DevSearch Q, GroupFilter F, const Tile* tiles,
                             unsigned int* bits) {
  const int lane = threadIdx.x & 31;
  const unsigned int total = *F.nlist;
  const int g = S.grp_g;
  unsigned int seen = 0;
  for (unsigned int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < total;
       e += (gridDim.x * blockDim.x) >> 5) {
    const uint2 en = F.list[e];
    const unsigned int tk = group_code_tile(en.x);
    const Tile T = tiles[tk];
    if (group_tile_dense(T, g, F.tcount[tk])) continue;
    const GroupPair p = group_code_pair(en.x, T, kGrpFan * g);
    unsigned int* out = bits + (size_t)tk * kLbLags * kLbWords;
    for (unsigned int mask = en.y; mask; mask &= mask - 1u) {
      const int b = __ffs(mask) - 1;
      const int64_t ia = (int64_t)(p.I * kGrpFan + (b >> 2)) * g;
      const int64_t ja = (int64_t)(p.J * kGrpFan + (b & 3)) * g;
      for (int x = lane; x < g * g; x += 32) {
        const int64_t i = ia + x / g, j = ja + x % g, row = i - T.i0, lag = j - i - T.L0;
        if (row < 0 || row >= T.rows || j >= T.send || lag < 0 || lag >= kLbLags) continue;
        if (S.flat[i] || S.flat[j]) continue;
        atomicOr(&out[(size_t)(row >> 5) * kLbLags + lag], 1u << (row & 31));
        ++seen;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) seen += __shfl_xor_sync(0xffffffffu, seen, o);
  // the sweep counted every pair of a sparse tile as pruned
  if (lane == 0 && seen) atomicAdd(&Q.counters[kPrunedFast], 0ull - (unsigned long long)seen);
}

// Super-group records: the extremes over kGrpFan consecutive groups.
__global__ void k_group_sup(DevSeries S) {
  const int64_t G = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (G >= S.sup_n) return;
  const float4* src = S.grp + (int64_t)blockIdx.y * S.grp_n + G * kGrpFan;
  float4 r = src[0];
  for (int e = 1; e < kGrpFan; ++e) {
    const float4 x = src[e];
    r = make_float4(fminf(r.x, x.x), fmaxf(r.y, x.y), fmaxf(r.z, x.z), fminf(r.w, x.w));
  }
  S.sup[(int64_t)blockIdx.y * S.sup_n + G] = r;
}

// Segments in bit-reversed order (0, 16, 8, 24, 4, ...).
SegOrder seg_order(int d) {
  SegOrder o;
  int k = 0;
  for (int x = 0; x < 32; ++x) {
    int r = 0;
    for (int b = 0; b < 5; ++b) r |= ((x >> b) & 1) << (4 - b);
    if (r < d) o.seg[k++] = (unsigned char)r;
  }
  while (k < kGrpSlots) o.seg[k++] = 255;
  return o;
}

}  // namespace

void group_shape(int m, int64_t s, DevSeries* S) {
  S->grp_g = group_windows(m);
  S->grp_b = m / 32 > 4 ? m / 32 : 4;
  const int d = m / S->grp_b < 32 ? m / S->grp_b : 32;
  S->grp_d = (d + 3) / 4 * 4;
  const int64_t G = (int64_t)kGrpFan * S->grp_g;
  S->sup_n = (s + G - 1) / G + 2 * kSupRows;
  S->grp_n = S->sup_n * kGrpFan;
}

int launch_group_prep(const DevSeries& S, double* means, cudaStream_t st) {
  const int d = S.m / S.grp_b < 32 ? S.m / S.grp_b : 32;
  k_seg_means<<<(unsigned)((S.n + kThreads - 1) / kThreads), kThreads, 0, st>>>(S, S.grp_b, means);
  const dim3 grid((unsigned)((S.grp_n + kThreads - 1) / kThreads), (unsigned)S.grp_d);
  k_group_rec<<<grid, kThreads, 0, st>>>(S, means, seg_order(d));
  const dim3 sgrid((unsigned)((S.sup_n + kThreads - 1) / kThreads), (unsigned)S.grp_d);
  k_group_sup<<<sgrid, kThreads, 0, st>>>(S);
  return 3;
}

size_t group_items(int g, GroupFilter* F) {
  // rows of a tile touch at most kLbRows / G + 1 super-groups; the lags from
  // one row group at most (kLbLags + G - 2) / G + 2 column groups
  const int G = kGrpFan * g, rows = kLbRows / G + 1, cols = (kLbLags + G - 2) / G + 2;
  F->nib = (rows + kSupRows - 1) / kSupRows;
  F->nw = (cols + kSupRows - 1 + kSupCols - 1) / kSupCols;
  return (size_t)rows * cols;
}

namespace {
template <bool ED>
void run_group(const DevSeries& S, const DevSearch& Q, const GroupFilter& F, const Tile* tiles,
               int ntiles, int num_sms, cudaStream_t st) {
  const unsigned int items = (unsigned int)ntiles * (unsigned)(F.nib * F.nw);
  k_group_super<ED><<<(items + kThreads / 32 - 1) / (kThreads / 32), kThreads, 0, st>>>(
      S, Q, F, tiles, items);
  k_group<ED><<<num_sms * 8, kThreads, 0, st>>>(S, Q, F, tiles);
}
}  // namespace

void launch_group_probe(const DevSeries& S, const DevSearch& Q, const GroupFilter& F,
                        const Tile* tiles, int ntiles, cudaStream_t st) {
  k_group_probe<false><<<kProbeSamples / (kThreads / 32), kThreads, 0, st>>>(S, Q, F, tiles, ntiles);
}

void launch_group(const DevSeries& S, const DevSearch& Q, const GroupFilter& F, const Tile* tiles,
                  int tile_begin, int tile_end, int num_sms, cudaStream_t st) {
  if (tile_end > tile_begin)
    run_group<false>(S, Q, F, tiles + tile_begin, tile_end - tile_begin, num_sms, st);
}

void launch_group_bits(const DevSeries& S, const DevSearch& Q, const GroupFilter& F,
                       const Tile* tiles, int tile_begin, int num_sms, unsigned int* bits,
                       cudaStream_t st) {
  k_group_bits<<<num_sms * 8, kThreads, 0, st>>>(S, Q, F, tiles + tile_begin, bits);
}

// ---- seeds of a large join ----
//
// The seeds are the kSeeds grid rows with the smallest ED to a later window
// (mp.cu).  Walking every diagonal for them (k_mp_seed) takes 0.2 ps per pair:
// 100 ms of the 1M-sample bench join once the sweep takes 30.  The group
// bound finds the same rows: with a cutoff c on ED^2, every pair below c lies
// in a group pair whose bound is at most c, and only those pairs are measured.
// c comes from a sample of row groups: each one's closest pair among its best
// group pair, and of these values the one that should leave a few times kSeeds
// rows below it.  Where the bound settles too little (it would cost more than
// walking the diagonals: quasi-periodic series) or a list overflows,
// *F.walk is set and k_mp_seed walks them after all.

namespace {

// Smallest group-pair bound of sampled row groups (one block each) over all
// later column groups, then the smallest ED^2 of the pairs of that group pair.
__global__ void __launch_bounds__(kThreads) k_seed_sample(DevSeries S, int64_t stride,
                                                          float* best_ed) {
  const int t = threadIdx.x, lane = t & 31;
  const int g = S.grp_g, m = S.m;
  const int64_t I = (int64_t)blockIdx.x * stride, n = S.grp_n;
  const int64_t ng = (S.s + g - 1) / g;
  __shared__ unsigned long long red[kThreads / 32];
  __shared__ float4 rec[kGrpSlots];
  if (t < S.grp_d) rec[t] = S.grp[t * n + I];
  __syncthreads();
  const float fb = (float)S.grp_b;
  float best = __int_as_float(0x7f800000);
  int64_t at = -1;
  for (int64_t J = (I * g + m + g - 1) / g + t; J < ng; J += kThreads) {
    float acc = 0.0f, unused = 0.0f;
    for (int s0 = 0; s0 < S.grp_d; s0 += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) group_terms<true>(rec[s0 + u], S.grp[(s0 + u) * n + J], acc, unused);
      if (fb * acc >= best) break;
    }
    if (fb * acc < best) {
      best = fb * acc;
      at = J;
    }
  }
  unsigned long long k = at < 0 ? ~0ull
                                : ((unsigned long long)__float_as_uint(best) << 32) | (unsigned int)at;
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, k, o);
    k = v < k ? v : k;
  }
  if (lane == 0) red[t >> 5] = k;
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < kThreads / 32; ++w) red[0] = red[w] < red[0] ? red[w] : red[0];
  }
  __syncthreads();
  k = red[0];
  __syncthreads();
  float ed = __int_as_float(0x7f800000);
  if (k != ~0ull) {
    const int64_t j0 = (int64_t)(k & 0xffffffffu) * g;
    for (int x = t >> 5; x < g * g; x += kThreads / 32) {
      const int64_t i = I * g + x / g, j = j0 + x % g;
      if (i >= S.s || j >= S.s || S.flat[i] || S.flat[j]) continue;
      const double mi = S.mu[i], si = S.isg[i], mj = S.mu[j], sj = S.isg[j];
      double d2 = 0.0;
      for (int q = lane; q < m; q += 32) {
        const double d = (S.a[i + q] - mi) * si - (S.a[j + q] - mj) * sj;
        d2 = fma(d, d, d2);
      }
      for (int o = 16; o > 0; o >>= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, o);
      ed = fminf(ed, (float)d2);
    }
  }
  if (lane == 0) red[t >> 5] = __float_as_uint(ed);
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < kThreads / 32; ++w) red[0] = red[w] < red[0] ? red[w] : red[0];
    best_ed[blockIdx.x] = __uint_as_float((unsigned int)red[0]);
  }
}

// cut = the rank-th smallest of the count sampled values (lowest index on
// ties), rounded up past the FP32 error of the bound.
__global__ void __launch_bounds__(1024) k_seed_cut(const float* v, int count, int rank, float* cut) {
  __shared__ float all[kSeedSamples];
  for (int x = threadIdx.x; x < count; x += blockDim.x) all[x] = v[x];
  __syncthreads();
  for (int x = threadIdx.x; x < count; x += blockDim.x) {
    const float mine = all[x];
    int below = 0;
#pragma unroll 8
    for (int y = 0; y < count; ++y) below += all[y] < mine || (all[y] == mine && y < x) ? 1 : 0;
    if (below == rank) *cut = mine * (1.0f + 1.0f / 4096.0f) + 1e-6f;
  }
}

// Exact ED^2 (FP64 centered dot product) of the grid rows of the surviving
// group pairs against their column windows, one warp per row and column
// group; the row's key takes the smallest, in the format of k_mp.
template <int G>
__global__ void __launch_bounds__(kThreads) k_seed_exact(DevSeries S, GroupFilter F,
                                                         const Tile* tiles, unsigned int budget,
                                                         unsigned long long* keys) {
  const int lane = threadIdx.x & 31;
  const unsigned int total = *F.nlist;
  // too many group pairs, or some were dropped: the diagonals are walked instead
  if (group_off(F, true, seed_share(G)) || total > F.list_cap || *F.nsup > F.sup_cap || *F.tcount > budget) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *F.walk = 1u;
    return;
  }
  const int m = S.m;
  const double two_m = 2.0 * m;
  for (unsigned int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < total;
       e += (gridDim.x * blockDim.x) >> 5) {
    const uint2 en = F.list[e];
    const Tile T = tiles[group_code_tile(en.x)];
    const GroupPair p = group_code_pair(en.x, T, kGrpFan * G);
    for (unsigned int mask = en.y; mask; mask &= mask - 1u) {
      const int b = __ffs(mask) - 1;
      const int ia = (p.I * kGrpFan + (b >> 2)) * G, j0 = (p.J * kGrpFan + (b & 3)) * G;
      // rows of the series' grid (a single series starts at window 0)
      for (int i = (ia + kSeedGrid - 1) / kSeedGrid * kSeedGrid; i < ia + G; i += kSeedGrid) {
        if (i < T.i0 || i >= T.i0 + T.rows || S.flat[i]) continue;
        const double mi = S.mu[i];
        double c[G], mj[G];
#pragma unroll
        for (int x = 0; x < G; ++x) {
          c[x] = 0.0;
          mj[x] = S.mu[j0 + x < T.send ? j0 + x : T.send - 1];
        }
        for (int k = lane; k < m; k += 32) {
          const double ai = S.a[i + k] - mi;
#pragma unroll
          for (int x = 0; x < G; ++x) {
            const int64_t q = (int64_t)j0 + x + k;
            c[x] = fma(ai, S.a[q < S.n ? q : S.n - 1] - mj[x], c[x]);
          }
        }
#pragma unroll
        for (int x = 0; x < G; ++x)
          for (int o = 16; o > 0; o >>= 1) c[x] += __shfl_xor_sync(0xffffffffu, c[x], o);
        // lane x finishes pair x
        double mine = 0.0;
#pragma unroll
        for (int x = 0; x < G; ++x)
          if (lane == x) mine = c[x];
        const int j = j0 + lane, lag = j - i - T.L0;
        if (lane < G && j < T.send && lag >= 0 && lag < kLbLags && !S.flat[j]) {
          const double e2 = fmax(two_m - 2.0 * mine * S.isg[i] * S.isg[j], 0.0);
          const unsigned int hi = (unsigned int)__double2hiint(e2) & ~7u;
          atomicMin(&keys[i], ((unsigned long long)hi << 32) | (unsigned int)j);
        }
      }
    }
  }
}

}  // namespace

void launch_seed_groups(const DevSeries& S, GroupFilter F, const Tile* tiles, int ntiles,
                        int world, float* samples, unsigned long long* keys, int num_sms,
                        cudaStream_t st) {
  cudaMemsetAsync(keys, 0xff, (size_t)S.s * 8, st);
  cudaMemsetAsync(F.walk, 0, 12, st);  // and the probe's two words
  // one row group in `stride`, at most kSeedSamples; the rank that should
  // leave 4 kSeeds grid rows (of this shard) below the cutoff, at least 4 deep
  const int64_t ng = (S.s + S.grp_g - 1) / S.grp_g, rows = (S.s + kSeedGrid - 1) / kSeedGrid;
  int64_t stride = 64;
  while ((ng + stride - 1) / stride > kSeedSamples) stride *= 2;
  const int count = (int)((ng + stride - 1) / stride);
  int64_t rank = 4ll * kSeeds * world * count / rows;
  if (rank < 4) rank = 4;
  if (rank > count - 1) rank = count - 1;
  k_seed_sample<<<count, kThreads, 0, st>>>(S, stride, samples);
  k_seed_cut<<<1, 1024, 0, st>>>(samples, count, (int)rank, const_cast<float*>(F.cut));
  k_group_probe<true><<<kProbeSamples / (kThreads / 32), kThreads, 0, st>>>(S, DevSearch{}, F,
                                                                            tiles, ntiles);
  for (int b = 0; b < ntiles; b += kSeedSlab) {
    const int cnt = ntiles - b < kSeedSlab ? ntiles - b : kSeedSlab;
    cudaMemsetAsync(F.nsup, 0, 12, st);  // nsup, nlist and the group pair count
    run_group<true>(S, DevSearch{}, F, tiles + b, cnt, num_sms, st);
    // a group pair costs about 1000 (g = 8) or 300 (g = 4) warp instructions,
    // walking a diagonal about 0.23 per pair: the budget is half of that
    const double pairs = (double)cnt * kLbLags * kLbRows;
    const unsigned int budget = (unsigned int)(pairs / (S.grp_g == 8 ? 8192.0 : 4096.0));
    if (S.grp_g == 8)
      k_seed_exact<8><<<num_sms * 8, kThreads, 0, st>>>(S, F, tiles + b, budget, keys);
    else
      k_seed_exact<4><<<num_sms * 8, kThreads, 0, st>>>(S, F, tiles + b, budget, keys);
  }
}

}  // namespace dtwj
