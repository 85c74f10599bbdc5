// LB_Keogh's cumulative bound and the banded DTW of the join's queue, several
// pairs to a warp.
//
// A warp holds 32 / G slots of G lanes (one slot of the whole warp for wide
// bands), one pair each; a lane owns C
// consecutive diagonals of its pair's band (the layout of pairs.cu).  A row
// step costs a warp two shuffles, two shared loads and 3 C + 1 arithmetic
// instructions whatever it holds, and shuffles and shared loads issue at one
// warp per clock and SM (32 lanes/clk measured, against 128 for FFMA and 64
// for the three-input minimum), so one pair per warp with C = 2 to 4 spends
// as long on them as on the cells.  Narrow bands in slots share them.
//
// Pairs abandon at different rows, so the slots run at different rows of
// their pairs but always the same instructions: 2 C steps, then a vote; a slot
// that finished or abandoned takes the next pair from the queue, which the
// whole warp prepares (normalisation, cumulative bound), and the others go on
// where they were.  Three things keep the steps uniform:
//  - rows before 0 and past m - 1 run too.  The padding of q and t holds
//    multiples of kPadStep, equal on the diagonal d = 0 and at least kPadStep
//    apart off it, so a path enters at (0, 0) and leaves at (m - 1, m - 1) at
//    no cost and every other cell of the padding costs at least 1e18;
//  - the one cell past the band that a band cell can reach in its lane takes
//    a +inf mask, at the compile-time position HI = (2 w + 1) mod C (every cell
//    is masked when HI = -2); the lanes past the band read a sentinel for q,
//    so their cells are huge (slot_mask_ok says when that walls the band off);
//  - the best-so-far is read at the start of the steps and used at their end.
// The next pair's indices and window statistics are loaded one pair ahead.
//
// DTW stage of ECG-like joins on one B200, one pair per warp against slots:
// 16,384 samples, m = 512, w = 52: 220 -> 150 ms; 9,001, m = 200, w = 20: 17.5
// -> 9.2 ms; 14,000, m = 256, w = 13: 23.5 -> 13.3 ms; 24,000, m = 128, w = 7:
// 20.6 -> 10.8 ms (with slots alone, without the window table: 206, 12.7, 15.2
// and 12.8 ms).  64 registers (the compiler's choice at 256 threads) beat 117
// and 154 with fewer warps by 9 and 26 % at w = 52.
#pragma once
#include "dtwj_dev.cuh"

namespace dtwj {

constexpr float kPadStep = 1e9f;

struct SlotLayout {
  int qf, qb, tf, tb;  // padding before and after q and t
  int nc;              // cumulative-bound chunks of 8 rows
  int q_off, t_off, cb_off, total;
};

__host__ __device__ inline SlotLayout slot_layout(int m, int w, int C, int G) {
  SlotLayout l;
  const int g0 = w / C;
  l.qf = G;
  l.qb = g0 + 2 * C + 1;
  l.tf = w + 1;
  const int r = g0 + 3 * C + (G - 1) * (C - 1) - w;
  l.tb = r > 0 ? r + 2 : 2;
  l.nc = (m + 7) / 8;
  // q, t and the slots start on 16-byte boundaries
  l.q_off = (l.qf + 3) / 4 * 4;
  l.t_off = (l.q_off + m + l.qb + l.tf + 3) / 4 * 4;
  l.cb_off = l.t_off + m + l.tb;
  l.total = l.cb_off + l.nc + 2;
  l.total += ((20 - l.total % 32) + 32) % 32;
  return l;
}

// HI alone walls the band off: the last lane must be huge, by its sentinel
// (all its cells past the band) or by the mask (its last cell is cell HI),
// since lane 0 reads it as its left neighbour.
__host__ __device__ constexpr bool slot_mask_ok(int w, int C, int G) {
  return C * G == 2 * w + 2 || C * (G - 1) >= 2 * w + 1;
}
__host__ __device__ constexpr int slot_mask(int w, int C) {
  return (2 * w + 1) % C == 0 ? -1 : (2 * w + 1) % C;
}
// Fewest cells per lane covering band w with the single-cell mask; 0: none up to 8.
__host__ __device__ constexpr int slot_cells(int w, int G) {
  for (int C = 2; C <= 8; ++C)
    if (C * G >= 2 * w + 1 && slot_mask_ok(w, C, G)) return C;
  return 0;
}
// Whether some band picks (C, G) with mask HI (what is instantiated).
constexpr bool slot_mask_used(int C, int G, int HI) {
  for (int w = 0; w < 4 * G; ++w)
    if (slot_cells(w, G) == C && slot_mask(w, C) == HI) return true;
  return false;
}

constexpr size_t kSlotSmemPerWarp = 20 * 1024 + 512;
inline size_t slot_bytes(int m, int w, int C, int G) {
  return (size_t)(32 / G) * slot_layout(m, w, C, G).total * sizeof(float);
}

#ifdef __CUDACC__
namespace slots {

__device__ __forceinline__ float min3f(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// One row step of every lane, in place (band_step of pairs.cu).
template <int C, int G, int HI, typename TW>
__device__ __forceinline__ void step(float qr, const TW& tw, int g, const float (&pen)[C],
                                     float (&A)[C]) {
  const float left = __shfl_sync(0xffffffffu, A[C - 1], (g + G - 1) & (G - 1), G);
  {
    const float d = qr - tw(0);
    float x = fmaf(d, d, min3f(A[1], A[0], left));
    if (HI == -2 || HI == 0) x = fmaxf(x, pen[0]);
    A[0] = x;
  }
  const float right = __shfl_sync(0xffffffffu, A[0], (g + 1) & (G - 1), G);
#pragma unroll
  for (int c = 1; c < C; ++c) {
    const float up = (c + 1 < C) ? A[c + 1 < C ? c + 1 : 0] : right;
    const float d = qr - tw(c);
    float x = fmaf(d, d, min3f(up, A[c], A[c - 1]));
    if (HI == -2 || HI == c) x = fmaxf(x, pen[c]);
    A[c] = x;
  }
}

// A window read from one of its ends.
struct EndView {
  const float* v;
  int at, dir;
  __device__ float operator[](int k) const { return v[at + dir * k]; }
};

// The next pair of the queue, loaded ahead of its use (warp-uniform).
struct Next {
  int i, j, sr;
  double mi, si, mj, sj;
  bool have;
};

__device__ __forceinline__ Next fetch(const DevSeries& S, const DevSearch& Q, const int2* pairs,
                                      unsigned int total, bool table, int lane) {
  Next nx;
  unsigned int idx = 0;
  if (lane == 0) idx = atomicAdd(Q.queue_next, 1u);
  idx = __shfl_sync(0xffffffffu, idx, 0);
  nx.have = idx < total;
  nx.i = nx.j = nx.sr = 0;
  nx.mi = nx.si = nx.mj = nx.sj = 0.0;
  if (nx.have) {
    const int2 p = pairs[idx];
    nx.i = p.x;
    nx.j = p.y;
    if (p.x >= 0) {  // else taken out of the queue by LB_Petitjean
      nx.sr = Q.qser ? Q.qser[idx] : series_of(S, p.x);
      if (!table) {
        nx.mi = S.mu[p.x];
        nx.si = S.isg[p.x];
        nx.mj = S.mu[p.y];
        nx.sj = S.isg[p.y];
      }
    }
  }
  return nx;
}

// The whole warp prepares pair `nx` in one slot's memory: the z-normalised
// windows and the cumulative bound (suffix sums over chunks of 8 rows of the
// LB_Keogh terms of window i against the envelope of window j, the endpoint
// bound in place of the end rows' terms).  Returns the whole bound.  With the
// window table a lane copies four samples of each row at a time; without it
// the samples are normalised here, in FP64, as the table's were.
__device__ __forceinline__ float prepare_pair(const DevSeries& S, const Next& nx, bool table,
                                              float* q, float* t, float* cbc, int nc, int lane) {
  const int m = S.m;
  if (table) {
    const float* zi = S.zt + (size_t)nx.i * S.zm;
    const float* zj = S.zt + (size_t)nx.j * S.zm;
    const float* uj = S.zu + (size_t)nx.j * S.zm;
    const float* lj = S.zl + (size_t)nx.j * S.zm;
#pragma unroll 2
    for (int k0 = 0; k0 < m; k0 += 128) {
      const int k = k0 + 4 * lane;
      float sum = 0.0f;
      if (k < m) {
        const float4 a = *reinterpret_cast<const float4*>(zi + k);
        const float4 b = *reinterpret_cast<const float4*>(zj + k);
        const float4 u = *reinterpret_cast<const float4*>(uj + k);
        const float4 l = *reinterpret_cast<const float4*>(lj + k);
        if (k + 4 <= m) {
          *reinterpret_cast<float4*>(q + k) = a;
          *reinterpret_cast<float4*>(t + k) = b;
        } else {  // nothing past the last sample
          const float av[3] = {a.x, a.y, a.z}, bv[3] = {b.x, b.y, b.z};
#pragma unroll
          for (int x = 0; x < 3; ++x)
            if (k + x < m) {
              q[k + x] = av[x];
              t[k + x] = bv[x];
            }
        }
        // no terms at the window's ends: kBias = 3 samples there
        const int e = m - kBias - k;
        float d0 = max3f(a.x - u.x, l.x - a.x, 0.0f), d1 = max3f(a.y - u.y, l.y - a.y, 0.0f);
        float d2 = max3f(a.z - u.z, l.z - a.z, 0.0f), d3 = max3f(a.w - u.w, l.w - a.w, 0.0f);
        d0 = k > 0 && e > 0 ? d0 : 0.0f;
        d1 = k > 0 && e > 1 ? d1 : 0.0f;
        d2 = k > 0 && e > 2 ? d2 : 0.0f;
        d3 = e > 3 ? d3 : 0.0f;
        sum = fmaf(d0, d0, fmaf(d1, d1, fmaf(d2, d2, d3 * d3)));
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      if ((lane & 1) == 0 && k < m) cbc[k >> 3] = sum;
    }
  } else {
    const double* ai = S.a + nx.i;
    const double* aj = S.a + nx.j;
    const double* U = S.U + nx.j;
    const double* L = S.L + nx.j;
#pragma unroll 4
    for (int k0 = 0; k0 < m; k0 += 32) {
      const int k = k0 + lane;
      float term = 0.0f;
      if (k < m) {
        const float zq = (float)((ai[k] - nx.mi) * nx.si);
        q[k] = zq;
        t[k] = (float)((aj[k] - nx.mj) * nx.sj);
        const float u = (float)((U[k] - nx.mj) * nx.sj), l = (float)((L[k] - nx.mj) * nx.sj);
        const float d = max3f(zq - u, l - zq, 0.0f);
        if (k >= kBias && k < m - kBias) term = d * d;
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) term += __shfl_xor_sync(0xffffffffu, term, o);
      if ((lane & 7) == 0 && k < m) cbc[k >> 3] = term;
    }
  }
  __syncwarp();
  // the endpoint bound's two parts join the chunks of rows 0 and m - kBias
  // (one lane each; the right part is the left one of the reversed windows)
  float side = 0.0f;
  if (lane < 2) side = kim_side<float>(EndView{q, lane ? m - 1 : 0, lane ? -1 : 1},
                                       EndView{t, lane ? m - 1 : 0, lane ? -1 : 1});
  if (lane == 0) cbc[0] += side;
  __syncwarp();
  if (lane == 1) cbc[(m - kBias) >> 3] += side;
  __syncwarp();
  // lane l owns chunks [l per, l per + per): it suffix-sums its own from the
  // end, then adds the totals of the lanes above it
  const int per = (nc + 31) / 32;
  float run = 0.0f;
  for (int u = per - 1; u >= 0; --u) {
    const int x = lane * per + u;
    if (x >= nc) continue;
    run += cbc[x];
    cbc[x] = run;
  }
  float above = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_down_sync(0xffffffffu, above, o);
    if (lane + o < 32) above += v;
  }
  const float whole = __shfl_sync(0xffffffffu, above, 0);
  above -= run;
  for (int u = 0; u < per; ++u) {
    const int x = lane * per + u;
    if (x < nc) cbc[x] += above;
  }
  if (lane < 2) cbc[nc + lane] = 0.0f;
  __syncwarp();
  return whole;
}

// Blocks per SM asked of the compiler: 3 (80 registers) where that measured
// faster than its own choice of 64 with a few spills: wide bands (walk of 131k,
// m = 512, w = 103: 168 -> 141 ms, one pair per warp without slots and table
// 288) and few cells per lane (w = 7 and 13: 4 %); at 6 and 7 cells in slots 64
// registers win by 3 to 6 %.
constexpr int slot_blocks(int C, int G) { return G == 32 || C <= 4 ? 3 : 0; }

template <int C, int G, int HI>
__global__ void __launch_bounds__(256, slot_blocks(C, G)) k_dtw_slots(DevSeries S, DevSearch Q, const int2* pairs,
                                                   const unsigned int* npairs) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int NS = 32 / G;
  constexpr unsigned int kGroup = 0xffffffffu >> (32 - G);  // a slot's lanes
  // iterations between abandon checks: every 10 to 18 steps
  constexpr int kIters = C >= 5 ? 1 : (C == 4 ? 2 : (C == 3 ? 3 : 4));
  const int m = S.m, w = S.w;
  const int lane = threadIdx.x & 31, slot = lane / G, g = lane & (G - 1);
  const float INF = __int_as_float(0x7f800000);
  const SlotLayout lay = slot_layout(m, w, C, G);
  float* past_q = reinterpret_cast<float*>(smraw);  // 2 C sentinels
  float* warp_base = past_q + 16 + (size_t)(threadIdx.x >> 5) * NS * lay.total;
  float* q = warp_base + (size_t)slot * lay.total + lay.q_off;
  float* t = warp_base + (size_t)slot * lay.total + lay.t_off;
  const float* cbc = warp_base + (size_t)slot * lay.total + lay.cb_off;
  if (threadIdx.x < 16) past_q[threadIdx.x] = kPadQ;
  // padding (the interior is written per pair; zero until the first)
  for (int x = g; x < lay.qf; x += G) q[-1 - x] = kPadStep * (float)(x + 1);
  for (int x = g; x < lay.tf; x += G) t[-1 - x] = kPadStep * (float)(x + 1);
  for (int x = g; x < m; x += G) q[x] = t[x] = 0.0f;
  for (int x = g; x < lay.qb; x += G) q[m + x] = -kPadStep * (float)(x + 1);
  for (int x = g; x < lay.tb; x += G) t[m + x] = -kPadStep * (float)(x + 1);
  __syncthreads();
  const int d_lo = -w + g * C;
  const bool past = HI != -2 && d_lo > w;  // every cell of the lane is past the band
  const int g0 = w / C, c0 = w % C;
  const int tau_end = m - 1 + g0;  // lane g0 (cell c0 on d = 0) reaches row m - 1
  float pen[C], A[C], W[2 * C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    pen[c] = (d_lo + c <= w) ? 0.0f : INF;
    A[c] = INF;
  }
#pragma unroll
  for (int x = 0; x < 2 * C; ++x) W[x] = 0.0f;
  const unsigned int total = *npairs < Q.queue_cap ? *npairs : Q.queue_cap;
  const bool table = S.zt && *S.zready != 0u;
  unsigned int ncalls = 0, nabandoned = 0, nkeogh = 0;
  unsigned long long cells = 0;  // of this lane
  // the slot's pair
  bool active = false;
  int pi = 0, pj = 0, sr = 0, tau = 0, iter = 0;
  float thr = INF;
  const float* tb = t;
  const float* qb = past_q;
  const int qstep = past ? 0 : 2 * C;
  unsigned int idle = 0xffffffffu;  // lanes of the slots without a pair
  Next nx = fetch(S, Q, pairs, total, table, lane);
  for (;;) {
    while (idle && nx.have) {
      const int s = (__ffs(idle) - 1) / G;
      float* sb = warp_base + (size_t)s * lay.total;
      const Next cur = nx;
      nx = fetch(S, Q, pairs, total, table, lane);
      if (cur.i < 0) continue;
      const float now =
          __shfl_sync(0xffffffffu, prune_threshold_now(Q.bsf2 + cur.sr, m), 0);
      const float whole = prepare_pair(S, cur, table, sb + lay.q_off, sb + lay.t_off, sb + lay.cb_off,
                                       lay.nc, lane);
      // the whole bound already exceeds the best-so-far: no DTW
      if (whole > now) {
        if (lane == 0) ++nkeogh;
        continue;
      }
      idle &= ~(kGroup << (s * G));
      if (slot == s) {
        active = true;
        pi = cur.i;
        pj = cur.j;
        sr = cur.sr;
        thr = now;
        tau = 0;
#pragma unroll
        for (int c = 0; c < C; ++c) A[c] = (d_lo + c == 0) ? 0.0f : INF;  // virtual row -g - 1
        const float* tg = t - g + d_lo;
#pragma unroll
        for (int x = 0; x < C - 1; ++x) W[x] = tg[x];
        tb = tg + C - 1;
        qb = past ? past_q : q - g;
      }
    }
    if (idle == 0xffffffffu) break;
    // 2 C steps (dtw_band of pairs.cu): q and the new values of t in
    // registers, t in a ring of 2 C
    const unsigned int bsf = *(volatile const unsigned int*)(Q.bsf2 + sr);
    float Qv[2 * C];
#pragma unroll
    for (int x = 0; x < C; ++x) W[C - 1 + x] = tb[x];
#pragma unroll
    for (int x = 0; x < 2 * C; ++x) Qv[x] = qb[x];
#pragma unroll
    for (int k = 0; k < C; ++k)
      step<C, G, HI>(Qv[k], [&W, k](int c) { return W[k + c]; }, g, pen, A);
#pragma unroll
    for (int x = 0; x < C; ++x) W[(2 * C - 1 + x) % (2 * C)] = tb[C + x];
#pragma unroll
    for (int k = 0; k < C; ++k)
      step<C, G, HI>(Qv[C + k], [&W, k](int c) { return W[(C + k + c) % (2 * C)]; }, g, pen, A);
    if (active) {
      tb += 2 * C;
      qb += qstep;
      tau += 2 * C;
    }
    const bool done = active && tau > tau_end;
    bool over = false;
    if (kIters == 1 || ++iter == kIters) {
      iter = 0;
      thr = fminf(thr, prune_threshold(bsf, m));
      float fm = A[0];
#pragma unroll
      for (int c = 1; c < C; ++c) fm = fminf(fm, A[c]);
      // The bound's terms belong to rows, and a path's last cell on the lanes'
      // frontier lies on the latest row of its lane: rows fall by at most one
      // per lane, so the path can only leave from there.  Every later row is
      // still ahead, also those within w of it.
      int idx = tau - g;
      idx = idx < 0 ? 0 : (idx + 7) >> 3;
      over = fm + cbc[idx < lay.nc ? idx : lay.nc] > thr;
    }
    const unsigned int ob = __ballot_sync(0xffffffffu, over) >> (slot * G);
    const bool ab = active && !done && (ob & kGroup) == kGroup;
    const unsigned int ended = __ballot_sync(0xffffffffu, done || ab);
    if (ended) {
      float d2 = INF;
      if (__any_sync(0xffffffffu, done)) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (c == c0) d2 = A[c];
        d2 = __shfl_sync(0xffffffffu, d2, g0, G);
      }
      if (done || ab) {
        // cells swept: rows [0, rows) of each diagonal the lane owns
        const int rows = tau - g < 0 ? 0 : (tau - g > m ? m : tau - g);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int d = d_lo + c;
          const int lo = d < 0 ? -d : 0, hi = rows < m - d ? rows : m - d;
          if (d <= w && hi > lo) cells += (unsigned int)(hi - lo);
        }
      }
      if ((done || ab) && g == 0) {
        ++ncalls;
        if (ab) {
          ++nabandoned;
        } else if (d2 <= prune_threshold_now(Q.bsf2 + sr, m)) {
          atomicMin(Q.bsf2 + sr, __float_as_uint(d2));
          const unsigned int at = atomicAdd(Q.cand_count, 1u);
          if (at < Q.cand_cap) {
            Candidate cd;
            cd.i = pi;
            cd.j = pj;
            cd.d2 = d2;
            cd.series = sr;
            Q.cand[at] = cd;
          }
        }
      }
      if (done || ab) {
        // an empty slot steps in place until it gets a pair
        active = false;
        tb = t;
        qb = past_q;
      }
      idle |= ended;
    }
  }
  unsigned long long nc = ncalls, na = nabandoned, nk = nkeogh;
  for (int o = 16; o > 0; o >>= 1) {
    nc += __shfl_xor_sync(0xffffffffu, nc, o);
    na += __shfl_xor_sync(0xffffffffu, na, o);
    nk += __shfl_xor_sync(0xffffffffu, nk, o);
    cells += __shfl_xor_sync(0xffffffffu, cells, o);
  }
  if (lane == 0) {
    if (nc) atomicAdd(&Q.counters[kDtwCalls], nc);
    if (na) atomicAdd(&Q.counters[kDtwAbandoned], na);
    if (nk) atomicAdd(&Q.counters[kPrunedKeogh], nk);
    if (cells) atomicAdd(&Q.counters[kDtwCells], cells);
  }
}

template <int C, int G, int HI>
void launch(const DevSeries& S, const DevSearch& Q, const int2* pairs, const unsigned int* npairs,
            int num_sms, cudaStream_t st, int warps) {
  if (warps <= 0) warps = 2;
  auto kern = k_dtw_slots<C, G, HI>;
  const size_t per_warp = slot_bytes(S.m, S.w, C, G);
  while (warps > 1 && warps * per_warp > 100 * 1024) warps /= 2;
  const size_t bytes = 64 + warps * per_warp;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, bytes);
  if (per_sm < 1) per_sm = 1;
  kern<<<num_sms * per_sm, 32 * warps, bytes, st>>>(S, Q, pairs, npairs);
}

// The mask HI of (w, C) where it walls the band off, else every cell masked.
template <int C, int G, int HI>
bool launch_hi(const DevSeries& S, const DevSearch& Q, const int2* pairs,
               const unsigned int* npairs, int num_sms, cudaStream_t st, int warps) {
  if constexpr (HI >= C) {
    return false;
  } else {
    if constexpr (slot_mask_used(C, G, HI)) {
      if (slot_mask_ok(S.w, C, G) && slot_mask(S.w, C) == HI) {
        launch<C, G, HI>(S, Q, pairs, npairs, num_sms, st, warps);
        return true;
      }
    }
    return launch_hi<C, G, HI == -1 ? 1 : HI + 1>(S, Q, pairs, npairs, num_sms, st, warps);
  }
}

template <int G, int C>
bool launch_c(int cells, const DevSeries& S, const DevSearch& Q, const int2* pairs,
              const unsigned int* npairs, int num_sms, cudaStream_t st, int warps) {
  if constexpr (C > 8) {
    return false;
  } else {
    if (cells != C)
      return launch_c<G, C + 1>(cells, S, Q, pairs, npairs, num_sms, st, warps);
    if (!launch_hi<C, G, -1>(S, Q, pairs, npairs, num_sms, st, warps))
      launch<C, G, -2>(S, Q, pairs, npairs, num_sms, st, warps);
    return true;
  }
}

}  // namespace slots
#endif
}  // namespace dtwj
