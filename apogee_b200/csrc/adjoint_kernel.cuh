// Adjoint of the fused filter's peak values at fixed lags.
//
// A reported peak of pair (d, t) in bin b is z = sum_f D[d,f] conj(H[t,f]) W^(f k)
// with W = exp(2 pi i / n) and k its lag.  With g the upstream gradient of z in
// torch's convention (dL/dRe z + i dL/dIm z), z is holomorphic in D and
// antiholomorphic in H, so with V_dt[f] = sum_b conj(g_dtb) W^(f k_dtb)
//
//   grad_D[d, f] = sum_t conj(V_dt[f]) H[t, f]
//   grad_H[t, f] = sum_d      V_dt[f]  D[d, f]
//
// V is the transform of a sequence with one entry per peak.  A thread owns
// the 16 frequencies f0 + j n/16, for which W^(f k) = W^(f0 k) e^(2 pi i j k/16):
// the entries are summed into 16 buckets by k mod 16, each entry costing one
// twiddled add whatever the number of frequencies, and one 16-point transform
// of the buckets gives V at all 16.  (Evaluating every entry at every
// frequency, two frequencies per twiddle, is about five times the arithmetic
// at 16 entries per pair.)
//
// One kernel serves both gradients: "own" rows are the ones written (d for
// grad_D, t for grad_H), "other" rows are summed over.  A CTA covers F =
// min(n/16, 256) values of f0 for 256/F own rows.  Entries are staged in
// rounds: a warp sorts one (own, other) row's entries by bucket, then the CTA
// tabulates W^(l k) for the 32 lanes l and conj(g) W^((F x + 32 a) k) for its
// groups a of 32 lanes (W^m = hi[m >> lo_bits] (1 + lo[m & mask]), FP64-built
// halves; the second is a root less one, so it adds no rounding of its own),
// so the inner loop is two shared-memory reads (the second a broadcast) and
// four FMAs per entry.  Rows without a peak are
// skipped.  Where the summed rows split over many CTAs, clusters of ADJ_CLUSTER
// of them add up their sums through distributed shared memory first: 291 atomic
// additions in a row to one output (3 x 872 pairs at n = 2048) doubled the
// gradient's rounding.  The lags are the forward pass's argmax lags; nothing of the
// correlation series is stored.  Runs with little to sum take adjoint_direct.cuh.
#pragma once
#include <cooperative_groups.h>
#include <cstdint>
#include "fft_radix.cuh"

namespace mfb {

constexpr int ADJ_THREADS = 256;
constexpr int ADJ_R = 16;              // frequencies per thread = buckets
constexpr int ADJ_CHUNK = 32;          // entries of one (own, other) row sorted at a time
constexpr int ADJ_TAB = 40960;         // bytes of staged twiddles per round
constexpr int ADJ_ITEMS = 1024;        // (own, other, chunk) lists per round
constexpr int ADJ_CLUSTER = 8;         // CTAs of one tile that add up before the atomics
static_assert(ADJ_R * ADJ_THREADS * sizeof(float2) <= ADJ_TAB, "a CTA's sums fit the staged twiddles");

struct AdjArgs {
  const float2 *src;      // other rows [other][n]: templates (grad_D) or data (grad_H)
  const int64_t *idx;     // [nd][nt][nb] lags; < 0 where no peak was reported
  const float2 *gz;       // [nd][nt][nb] upstream gradient of the peak value
  float2 *out;            // [own][n]
  int n, nd, nt, nb;
  int own, other;
  int fblk, slots;        // f0 values and own rows per CTA (fblk * slots = 256)
  int fx;                 // blocks of fblk f0 values
  int chunk;              // entries per list, <= ADJ_CHUNK
  int chunks;             // lists per (own, other) row: ceil(nb / chunk)
  int rows_per_round;     // other rows per round when chunks == 1, else 1
  int lists_per_round;    // lists of one row per round when chunks > 1, else 1
  int other_per_split;    // other rows per blockIdx.y
  int accumulate;         // 1: atomicAdd into a zeroed out (other split over blockIdx.y)
  int lsh, ash;           // log2 of the lane and group values per entry
  int clusters;           // 1: blockIdx.y in clusters of ADJ_CLUSTER
  const float2 *tw_hi, *tw_lo;
  int lo_bits, hi_count;
};

// Bytes of staged twiddles per entry: min(fblk, 32) lane values, one value
// per group of 32 f0.
__host__ __device__ constexpr int adj_entry_bytes(int fblk) {
  return 8 * ((fblk < 32 ? fblk : 32) + (fblk + 31) / 32);
}

template <bool GRAD_DATA>
__global__ void __launch_bounds__(ADJ_THREADS, 2) adjoint_kernel(const AdjArgs a) {
  extern __shared__ __align__(16) unsigned char adj_smem[];
  const int L = 1 << a.lsh, A = 1 << a.ash;
  const int per_item = a.chunk;
  const int cap = ADJ_TAB / adj_entry_bytes(a.fblk);          // entries per round
  float2 *lane_tw = reinterpret_cast<float2 *>(adj_smem);      // [cap][L]
  float2 *group_tw = lane_tw + cap * L;                        // [cap][A]
  float2 *s_g = group_tw + cap * A;                            // [cap] conj(g), sorted
  int *s_k = reinterpret_cast<int *>(s_g + cap);               // [cap] lags, sorted
  float2 *s_hi = reinterpret_cast<float2 *>(                   // twiddle halves
      (reinterpret_cast<uintptr_t>(s_k + cap) + 15) & ~uintptr_t(15));
  float2 *s_lo = s_hi + a.hi_count;
  uint4 *s_end = reinterpret_cast<uint4 *>(                    // [items] bucket ends, one byte each
      (reinterpret_cast<uintptr_t>(s_lo + (1 << a.lo_bits)) + 15) & ~uintptr_t(15));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int fb = blockIdx.x % a.fx, oc = blockIdx.x / a.fx;
  const int i = tid & (a.fblk - 1), slot = tid / a.fblk;       // fblk is a power of two
  const int l = i & 31, grp = i >> 5;
  const int own_row = oc * a.slots + slot;
  const int sixteenth = a.n >> 4;
  const int f0 = fb * a.fblk + i;
  const int ob = blockIdx.y * a.other_per_split;
  const int oe = min(a.other, ob + a.other_per_split);
  const unsigned mask_n = (unsigned)a.n - 1u;
  const unsigned lo_mask = (1u << a.lo_bits) - 1u;
  const bool live = own_row < a.own;
  for (int x = tid; x < a.hi_count; x += ADJ_THREADS) s_hi[x] = a.tw_hi[x];
  for (int x = tid; x <= (int)lo_mask; x += ADJ_THREADS) s_lo[x] = a.tw_lo[x];
  auto root = [&](unsigned m) {   // W^(m mod n)
    m &= mask_n;
    const float2 h = s_hi[m >> a.lo_bits], w = s_lo[m & lo_mask];
    return cf{fmaf(h.x, w.x, fmaf(-h.y, w.y, h.x)), fmaf(h.x, w.y, fmaf(h.y, w.x, h.y))};
  };

  cf acc[ADJ_R];
#pragma unroll
  for (int j = 0; j < ADJ_R; j++) acc[j] = {0.f, 0.f};

  for (int o0 = ob; o0 < oe; o0 += a.rows_per_round) {
    const int rr = min(a.rows_per_round, oe - o0);
    cf S[ADJ_R];
    int seen = 0;                       // entries of the row so far (rows of several rounds)
    for (int c0 = 0; c0 < a.chunks; c0 += a.lists_per_round) {
      const int lc = min(a.lists_per_round, a.chunks - c0);
      const int items = rr * lc * a.slots;             // list (o, chunk, slot): slot fastest
      __syncthreads();                                 // the previous round's readers are done
      // ---- each warp sorts whole lists by k mod 16 --------------------------------
      for (int it = warp; it < items; it += ADJ_THREADS / 32) {
        const int s = it % a.slots, oq = it / a.slots;
        const int cl = oq % lc, o = o0 + oq / lc, mine = oc * a.slots + s;
        const int b = (c0 + cl) * a.chunk + lane;
        int k = -1;
        float2 g = make_float2(0.f, 0.f);
        if (lane < a.chunk && b < a.nb && mine < a.own) {
          const int d = GRAD_DATA ? mine : o, t = GRAD_DATA ? o : mine;
          const long long at = ((long long)d * a.nt + t) * a.nb + b;
          const long long kk = a.idx[at];
          if (kk >= 0) {
            k = (int)(kk & mask_n);
            g = a.gz[at];
            g.y = -g.y;
          }
        }
        const int c = k >= 0 ? (k & (ADJ_R - 1)) : ADJ_R;
        unsigned ends[4] = {0u, 0u, 0u, 0u};
        int before = 0, pos = 0;
#pragma unroll
        for (int q = 0; q < ADJ_R; q++) {
          const unsigned m = __ballot_sync(0xffffffffu, c == q);
          if (c == q) pos = before + __popc(m & ((1u << lane) - 1u));
          before += __popc(m);
          ends[q >> 2] |= (unsigned)before << (8 * (q & 3));
        }
        if (k >= 0) {
          s_k[it * per_item + pos] = k;
          s_g[it * per_item + pos] = g;
        }
        if (lane >= before && lane < a.chunk) s_k[it * per_item + lane] = -1;
        if (lane == 0) s_end[it] = make_uint4(ends[0], ends[1], ends[2], ends[3]);
      }
      __syncthreads();
      // ---- twiddle tables of every staged entry ------------------------------------
      for (int x = tid; x < items * per_item * L; x += ADJ_THREADS) {
        const int e = x >> a.lsh, j = x & (L - 1);
        const int k = s_k[e];
        if (k < 0) continue;
        const cf w = root((unsigned)j * (unsigned)k);
        lane_tw[x] = make_float2(w.x, w.y);
      }
      for (int x = tid; x < items * per_item * A; x += ADJ_THREADS) {
        const int e = x >> a.ash, j = x & (A - 1);
        const int k = s_k[e];
        if (k < 0) continue;
        const float2 g = s_g[e];
        const cf w = cmul(cf{g.x, g.y}, root((unsigned)(fb * a.fblk + 32 * j) * (unsigned)k));
        group_tw[x] = make_float2(w.x, w.y);
      }
      __syncthreads();
      // ---- V at this thread's 16 frequencies, times the other row ---------------------
      for (int ol = 0; ol < rr; ol++) {
        if (c0 == 0) {
          seen = 0;
#pragma unroll
          for (int j = 0; j < ADJ_R; j++) S[j] = {0.f, 0.f};
        }
        for (int cl = 0; cl < lc; cl++) {
          const int it = (ol * lc + cl) * a.slots + slot;
          const uint4 ends = s_end[it];
          const unsigned ew[4] = {ends.x, ends.y, ends.z, ends.w};
          const float2 *p1 = lane_tw + ((it * per_item) << a.lsh) + l;
          const float2 *p2 = group_tw + ((it * per_item) << a.ash) + grp;
          int e = 0;
#pragma unroll
          for (int q = 0; q < ADJ_R; q++) {
            const int end = (int)((ew[q >> 2] >> (8 * (q & 3))) & 255u);
#pragma unroll 1   // about one entry a bucket; unrolled: 128 us instead of 88 at n = 16384, 8 x 256
            for (; e < end; e++, p1 += L, p2 += A) {
              const float2 w = *p1, h = *p2;
              S[q].x = fmaf(w.x, h.x, fmaf(-w.y, h.y, S[q].x));
              S[q].y = fmaf(w.x, h.y, fmaf(w.y, h.x, S[q].y));
            }
          }
          seen += e;
        }
        if (c0 + lc < a.chunks || !live || seen == 0) continue;   // more of this row to come, or nothing
        dft16(S);
        const float2 *sp = a.src + (long long)(o0 + ol) * a.n + f0;
#pragma unroll
        for (int j = 0; j < ADJ_R; j++) {
          const float2 h = __ldg(sp + j * sixteenth);
          if (GRAD_DATA) {                // conj(V) * H
            acc[j].x = fmaf(S[j].x, h.x, fmaf(S[j].y, h.y, acc[j].x));
            acc[j].y = fmaf(S[j].x, h.y, fmaf(-S[j].y, h.x, acc[j].y));
          } else {                        // V * D
            acc[j].x = fmaf(S[j].x, h.x, fmaf(-S[j].y, h.y, acc[j].x));
            acc[j].y = fmaf(S[j].x, h.y, fmaf(S[j].y, h.x, acc[j].y));
          }
        }
      }
    }
  }
  float2 *op = a.out + (long long)own_row * a.n + f0;
  if (a.clusters) {       // each CTA adds up ADJ_R / ADJ_CLUSTER of the cluster's 16 frequencies
    const auto cluster = cooperative_groups::this_cluster();
    __syncthreads();      // the last round's readers are done
    float2 *sums = lane_tw;
#pragma unroll
    for (int j = 0; j < ADJ_R; j++) sums[j * ADJ_THREADS + tid] = make_float2(acc[j].x, acc[j].y);
    cluster.sync();
#pragma unroll
    for (int q = 0; q < ADJ_R / ADJ_CLUSTER; q++) {
      const int j = (int)cluster.block_rank() * (ADJ_R / ADJ_CLUSTER) + q;
      float2 v[ADJ_CLUSTER];
#pragma unroll
      for (int c = 0; c < ADJ_CLUSTER; c++) v[c] = cluster.map_shared_rank(sums, c)[j * ADJ_THREADS + tid];
#pragma unroll
      for (int h = 1; h < ADJ_CLUSTER; h *= 2) {
#pragma unroll
        for (int c = 0; c < ADJ_CLUSTER; c += 2 * h) {
          v[c].x += v[c + h].x;
          v[c].y += v[c + h].y;
        }
      }
      if (live) atomicAdd(op + j * sixteenth, v[0]);
    }
    cluster.sync();       // the other CTAs may still read this one's sums
    return;
  }
  if (!live) return;
#pragma unroll
  for (int j = 0; j < ADJ_R; j++) {
    const float2 v = make_float2(acc[j].x, acc[j].y);
    if (a.accumulate) atomicAdd(op + j * sixteenth, v);
    else op[j * sixteenth] = v;
  }
}

}  // namespace mfb
