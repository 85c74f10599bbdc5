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
// up), so only the evaluation rounds: each term is off by 2^-24 relative and
// the sum by (terms + 2) 2^-24 < 3e-6, inside the 1/512 the threshold keeps
// above the best-so-far.
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

// Means of the series and its envelope over [p, p + B), FP64: [3][n].
__global__ void k_seg_means(DevSeries S, int B, double* gm) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p + B > S.n) return;
  double sa = 0.0, su = 0.0, sl = 0.0;
  for (int k = 0; k < B; ++k) {
    sa += S.a[p + k];
    su += S.U[p + k];
    sl += S.L[p + k];
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
      const double q = (gm[p] - mu) * is;
      qlo = fmin(qlo, q);
      qhi = fmax(qhi, q);
      up = fmax(up, (gm[S.n + p] - mu) * is);
      lo = fmin(lo, (gm[2 * S.n + p] - mu) * is);
    }
    if (qlo <= qhi)
      rec = make_float4(__double2float_rd(qlo), __double2float_ru(qhi), __double2float_ru(up),
                        __double2float_rd(lo));
    else
      rec = make_float4(kFar, -kFar, -kFar, kFar);
  }
  S.grp[(int64_t)slot * S.grp_n + G] = rec;
}

// Both directions of one segment of a group pair.
__device__ __forceinline__ void group_terms(const float4 i, const float4 j, float& a1, float& a2) {
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
// consecutive row groups I; lane l takes the column group J = I + L0 / G1 + l
// (+ 32 w), the groups that hold lags of the tile.  The records of a slot are
// consecutive in memory: the J loads are coalesced and overlap from row to
// row, the I loads are broadcasts.  The slots are in an order that spreads
// the first ones over the window; the warp votes every four.
constexpr int kSupRows = 4;
__global__ void __launch_bounds__(kThreads) k_group_super(DevSeries S, DevSearch Q, GroupFilter F,
                                                          const Tile* tiles, unsigned int total) {
  const int lane = threadIdx.x & 31;
  const unsigned int item = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (item >= total) return;
  const unsigned int per = (unsigned int)(F.nib * F.nw);
  const unsigned int tk = item / per, rem = item - tk * per;
  const Tile T = tiles[tk];
  const int g = kGrpFan * S.grp_g;
  const int row0 = (int)(rem / (unsigned)F.nw) * kSupRows;   // relative to the tile's first
  const int col = (int)(rem % (unsigned)F.nw) * 32 + lane;   // relative to I + L0 / g
  const int I0 = T.i0 / g + row0;
  const int last_row = T.i0 + T.rows - 1;
  if ((int64_t)I0 * g > last_row) return;
  const int J0 = I0 + T.L0 / g + col;
  unsigned int alive = 0;
#pragma unroll
  for (int r = 0; r < kSupRows; ++r)
    if (group_pair_in_tile(T, g, I0 + r, J0 + r)) alive |= 1u << r;
  if (!__any_sync(0xffffffffu, alive != 0u)) return;
  const float thr = prune_threshold_now(Q.bsf2 + T.series, S.m);
  const float fb = (float)S.grp_b;
  const int64_t n = S.sup_n;
  // addresses past the last record repeat it (those group pairs are not
  // alive); the records run past the last row group by more than kSupRows
  const float4* pi = S.sup + I0;
  const float4* pj[kSupRows];
  float a1[kSupRows], a2[kSupRows];
#pragma unroll
  for (int r = 0; r < kSupRows; ++r) {
    pj[r] = S.sup + (J0 + r < n ? J0 + r : n - 1);
    a1[r] = a2[r] = 0.0f;
  }
#pragma unroll 1
  for (int s0 = 0; s0 < S.grp_d; s0 += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int r = 0; r < kSupRows; ++r) group_terms(pi[u * n + r], pj[r][u * n], a1[r], a2[r]);
    }
    pi += 4 * n;
#pragma unroll
    for (int r = 0; r < kSupRows; ++r) {
      pj[r] += 4 * n;
      if (fb * fmaxf(a1[r], a2[r]) > thr) alive &= ~(1u << r);
    }
    if (!__any_sync(0xffffffffu, alive != 0u)) return;
  }
#pragma unroll
  for (int r = 0; r < kSupRows; ++r) {
    const bool on = (alive >> r) & 1u;
    const unsigned int slot = append_slot(on, lane, F.nsup);
    if (on) F.sup[slot] = group_code(tk, row0 + r, col);
  }
}

// Second level: half a warp per surviving super-group pair, one lane per
// pair of its kGrpFan x kGrpFan groups.
__global__ void __launch_bounds__(kThreads) k_group(DevSeries S, DevSearch Q, GroupFilter F,
                                                    const Tile* tiles) {
  static_assert(kGrpFan == 4, "16 group pairs, half a warp");
  const int lane = threadIdx.x & 31, h = lane & 15;
  const unsigned int total = *F.nsup;
  const int g = S.grp_g, G = kGrpFan * g;
  const float fb = (float)S.grp_b;
  const int64_t n = S.grp_n;
  for (unsigned int e0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 2; e0 < total;
       e0 += ((gridDim.x * blockDim.x) >> 5) * 2) {
    const unsigned int e = e0 + (lane >> 4);
    const unsigned int code = F.sup[e < total ? e : total - 1];
    const unsigned int tk = group_code_tile(code);
    const Tile T = tiles[tk];
    const GroupPair p = group_code_pair(code, T, G);
    const int I = p.I * kGrpFan + (h >> 2), J = p.J * kGrpFan + (h & 3);
    bool alive = e < total && group_pair_in_tile(T, g, I, J);
    const float thr = prune_threshold_now(Q.bsf2 + T.series, S.m);
    const float4* pi = S.grp + (I < n ? I : n - 1);
    const float4* pj = S.grp + (J < n ? J : n - 1);
    float a1 = 0.0f, a2 = 0.0f;
#pragma unroll 1
    for (int s0 = 0; s0 < S.grp_d && __any_sync(0xffffffffu, alive); s0 += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) group_terms(pi[u * n], pj[u * n], a1, a2);
      pi += 4 * n;
      pj += 4 * n;
      alive = alive && !(fb * fmaxf(a1, a2) > thr);
    }
    const unsigned int mask = (__ballot_sync(0xffffffffu, alive) >> (lane & 16)) & 0xffffu;
    const bool on = h == 0 && mask != 0u;
    const unsigned int slot = append_slot(on, lane, F.nlist);
    if (on) {
      F.list[slot] = make_uint2(code, mask);
      atomicAdd(&F.tcount[tk], (unsigned int)__popc(mask));
    }
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
  F->nw = (cols + 31) / 32;
  return (size_t)rows * cols;
}

void launch_group(const DevSeries& S, const DevSearch& Q, const GroupFilter& F, const Tile* tiles,
                  int tile_begin, int tile_end, int num_sms, cudaStream_t st) {
  if (tile_end <= tile_begin) return;
  const unsigned int items = (unsigned int)(tile_end - tile_begin) * (unsigned)(F.nib * F.nw);
  k_group_super<<<(items + kThreads / 32 - 1) / (kThreads / 32), kThreads, 0, st>>>(
      S, Q, F, tiles + tile_begin, items);
  k_group<<<num_sms * 8, kThreads, 0, st>>>(S, Q, F, tiles + tile_begin);
}

void launch_group_bits(const DevSeries& S, const DevSearch& Q, const GroupFilter& F,
                       const Tile* tiles, int tile_begin, int num_sms, unsigned int* bits,
                       cudaStream_t st) {
  k_group_bits<<<num_sms * 8, kThreads, 0, st>>>(S, Q, F, tiles + tile_begin, bits);
}

}  // namespace dtwj
