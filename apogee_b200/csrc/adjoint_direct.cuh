// Adjoint of the peak values for runs with little to sum: every entry evaluated at
// every frequency, the formulas of adjoint_kernel.cuh without its buckets.
//
// A thread owns frequencies f and f + n/2, whose twiddles differ by (-1)^k, of OC own
// rows; a CTA stages the (lag, gradient) entries of its rows in shared memory and reads
// them as broadcasts, W^m = hi[m >> lo_bits] lo[m & mask].  An entry costs a twiddled
// product at each frequency where the buckets cost one per 16, but nothing is sorted,
// tabulated or transformed first and all n frequencies of few rows are worked on at
// once, so it is the faster form while launch and staging latency bound the run, and
// with one entry per pair (which the buckets' 16-point transform cannot win back).
// adjoint_direct (mfb_api.cu) has the rule and both sides' times.
//
// Rounding: the rule leaves a CTA 16 summed rows at most, more than 16 entries of a pair
// are summed in two chains, and where the summed rows split over more than ADJD_ATOMICS
// CTAs clusters of them add up their sums before the atomics: relative 2-norm errors of
// 0.5 to 1.8e-7 over 444 shapes (the buckets: 0.4 to 2.2e-7).  Without that 512 and 1024 rows gave 2.8
// to 4.1e-7 against the buckets' 1.2 to 1.7e-7.
#pragma once
#include <climits>
#include "adjoint_kernel.cuh"

namespace mfb {

constexpr int ADJD_CAP = 2048;      // staged entries per round
constexpr int ADJD_TW = 1024;       // entries of each twiddle half-table (n <= 2^20)
constexpr int ADJD_ROWS = 16;       // rows a CTA sums, at most
constexpr int ADJD_ATOMICS = 16;    // splits added by atomics alone, at most

struct AdjDirectArgs {
  const float2 *src;                // as in AdjArgs
  const int64_t *idx;
  const float2 *gz;
  float2 *out;
  int n, nd, nt, nb, own, other;
  int rows_per_round, bins_per_round;
  int other_per_split;              // other rows per blockIdx.z
  int accumulate, clusters;         // clusters: blockIdx.z in clusters of ADJ_CLUSTER (OC = 1)
  const float2 *tw_hi, *tw_lo;
  int lo_bits, hi_count;
};

template <int OC, bool GRAD_DATA>
__global__ void __launch_bounds__(ADJ_THREADS, OC == 8 ? 4 : 5) adjoint_direct_kernel(const AdjDirectArgs a) {
  __shared__ float2 s_hi[ADJD_TW], s_lo[ADJD_TW];
  __shared__ int s_k[ADJD_CAP];
  __shared__ float2 s_g[ADJD_CAP];
  const int half = a.n >> 1, tid = threadIdx.x;
  const int f = blockIdx.x * ADJ_THREADS + tid;
  const int j0 = blockIdx.y * OC;
  const int ob = blockIdx.z * a.other_per_split;
  const int oe = min(a.other, ob + a.other_per_split);
  const unsigned mask_n = (unsigned)a.n - 1u, lo_mask = (1u << a.lo_bits) - 1u;
  for (int i = tid; i < a.hi_count; i += ADJ_THREADS) s_hi[i] = a.tw_hi[i];
  for (int i = tid; i <= (int)lo_mask; i += ADJ_THREADS) s_lo[i] = a.tw_lo[i];
  cf acc0[OC], acc1[OC];
#pragma unroll
  for (int j = 0; j < OC; j++) acc0[j] = acc1[j] = cf{0.f, 0.f};

  for (int o0 = ob; o0 < oe; o0 += a.rows_per_round) {
    const int rr = min(a.rows_per_round, oe - o0);
    for (int b0 = 0; b0 < a.nb; b0 += a.bins_per_round) {
      const int bc = min(a.bins_per_round, a.nb - b0);
      const int per_row = OC * bc, total = rr * per_row;
      __syncthreads();   // the previous round's readers are done (and the tables are in)
      for (int e = tid; e < total; e += ADJ_THREADS) {
        const int ol = e / per_row, rem = e - ol * per_row;
        const int jj = rem / bc, bl = rem - jj * bc;
        const int own_row = j0 + jj;
        int k = INT_MIN;               // no peak: W^0 times a zero
        float2 g = make_float2(0.f, 0.f);
        if (own_row < a.own) {
          const int o = o0 + ol;
          const int d = GRAD_DATA ? own_row : o, t = GRAD_DATA ? o : own_row;
          const long long i = ((long long)d * a.nt + t) * a.nb + b0 + bl;
          const long long kk = a.idx[i];
          if (kk >= 0) {
            k = (int)(kk & mask_n);
            g = a.gz[i];
            if (!GRAD_DATA) g.y = -g.y;   // conj(g)
          }
        }
        s_k[e] = k;
        s_g[e] = g;
      }
      __syncthreads();
      if (f >= half) continue;
      for (int ol = 0; ol < rr; ol++) {
        const float2 *sp = a.src + (long long)(o0 + ol) * a.n;
        const float2 s0 = __ldg(sp + f), s1 = __ldg(sp + f + half);
#pragma unroll
        for (int jj = 0; jj < OC; jj++) {
          const int eb = (ol * OC + jj) * bc;
          int dead = -1;               // negative while every entry is
          auto term = [&](int e, cf &u0, cf &u1) {
            const int k = s_k[e];
            const float2 g = s_g[e];
            dead &= k;
            const unsigned m = ((unsigned)f * (unsigned)k) & mask_n;
            const float2 wh = s_hi[m >> a.lo_bits], wl = s_lo[m & lo_mask];
            const float wr = fmaf(wh.x, wl.x, -wh.y * wl.y);
            const float wi = fmaf(wh.x, wl.y, wh.y * wl.x);
            float tr, ti;
            if (GRAD_DATA) {           // g * conj(W^(fk))
              tr = fmaf(g.x, wr, g.y * wi);
              ti = fmaf(g.y, wr, -g.x * wi);
            } else {                   // conj(g) * W^(fk)
              tr = fmaf(g.x, wr, -g.y * wi);
              ti = fmaf(g.x, wi, g.y * wr);
            }
            const float sgn = (k & 1) ? -1.f : 1.f;   // W^((f + n/2) k) = (-1)^k W^(fk)
            u0.x += tr;
            u0.y += ti;
            u1.x = fmaf(sgn, tr, u1.x);
            u1.y = fmaf(sgn, ti, u1.y);
          };
          cf u0 = {0.f, 0.f}, u1 = {0.f, 0.f};
          int bl = 0;
          if (bc > 16) {               // two chains
            cf v0 = {0.f, 0.f}, v1 = {0.f, 0.f};
            const int h = bc >> 1;
            for (; bl < h; bl++) {
              term(eb + bl, u0, u1);
              term(eb + h + bl, v0, v1);
            }
            bl += h;
            u0.x += v0.x; u0.y += v0.y;
            u1.x += v1.x; u1.y += v1.y;
          }
          for (; bl < bc; bl++) term(eb + bl, u0, u1);
          // no peak: the row (were it NaN) adds nothing
          const float2 h0 = dead < 0 ? make_float2(0.f, 0.f) : s0, h1 = dead < 0 ? make_float2(0.f, 0.f) : s1;
          acc0[jj].x = fmaf(h0.x, u0.x, fmaf(-h0.y, u0.y, acc0[jj].x));
          acc0[jj].y = fmaf(h0.x, u0.y, fmaf(h0.y, u0.x, acc0[jj].y));
          acc1[jj].x = fmaf(h1.x, u1.x, fmaf(-h1.y, u1.y, acc1[jj].x));
          acc1[jj].y = fmaf(h1.x, u1.y, fmaf(h1.y, u1.x, acc1[jj].y));
        }
      }
    }
  }
  if constexpr (OC == 1) {
    if (a.clusters) {       // each CTA adds up a part of the cluster's 512 sums
      const auto cluster = cooperative_groups::this_cluster();
      __syncthreads();      // the last round's readers are done
      float2 *sums = s_g;
      sums[tid] = make_float2(acc0[0].x, acc0[0].y);
      sums[ADJ_THREADS + tid] = make_float2(acc1[0].x, acc1[0].y);
      cluster.sync();
      constexpr int PART = 2 * ADJ_THREADS / ADJ_CLUSTER;
      if (tid < PART) {
        const int e = (int)cluster.block_rank() * PART + tid;
        float2 v[ADJ_CLUSTER];
#pragma unroll
        for (int c = 0; c < ADJ_CLUSTER; c++) v[c] = cluster.map_shared_rank(sums, c)[e];
#pragma unroll
        for (int h = 1; h < ADJ_CLUSTER; h *= 2)
#pragma unroll
          for (int c = 0; c < ADJ_CLUSTER; c += 2 * h) {
            v[c].x += v[c + h].x;
            v[c].y += v[c + h].y;
          }
        const int fe = blockIdx.x * ADJ_THREADS + (e & (ADJ_THREADS - 1));
        if (fe < half)
          atomicAdd(a.out + (long long)j0 * a.n + fe + (e >= ADJ_THREADS ? half : 0), v[0]);
      }
      cluster.sync();       // the other CTAs may still read this one's sums
      return;
    }
  }
  if (f >= half) return;
#pragma unroll
  for (int jj = 0; jj < OC; jj++) {
    if (j0 + jj >= a.own) break;
    float2 *op = a.out + (long long)(j0 + jj) * a.n + f;
    const float2 v0 = make_float2(acc0[jj].x, acc0[jj].y), v1 = make_float2(acc1[jj].x, acc1[jj].y);
    if (a.accumulate) {
      atomicAdd(op, v0);
      atomicAdd(op + half, v1);
    } else {
      op[0] = v0;
      op[half] = v1;
    }
  }
}

}  // namespace mfb
