// Fused matched filter at n = 4096 with two pairs per thread (packed FP32x2).
//
// Same pair transform as flat_kernel<4096, MODE_PEAKS> (conjugate product ->
// unnormalised inverse FFT -> per-bin argmax, src/balanced-inl.h:1102-1113 in
// the reference), restructured for sm_100a's packed FP32 instructions: every
// thread carries the same butterfly of TWO pairs at once, lane A and lane B of
// float2 registers (X = (re_A, re_B), Y = (im_A, im_B)), so each add, multiply
// or FMA of the radix-16 Stockham passes is one FADD2 / FMUL2 / FFMA2 for both
// pairs.  The butterflies' operations, their order and their roundings are
// those of the scalar kernel; the packed form halves the FP32 instructions
// and the barriers per pair.
//
// Layout:
//  * a CTA of 256 threads = one pair slot of T = n/16 threads, two pairs per
//    item (pairs 2i and 2i+1 of the dense block or of the row list);
//  * the exchange buffer holds float4 records (re_A, re_B, im_A, im_B) with
//    the scalar kernel's padding (one record per 16), 69.6 KB, so two CTAs fit
//    on an SM;
//  * inter-pass twiddles are float4 (wr, wr, wi, wi) -- the same FP64-built
//    values as the scalar tables, duplicated for the two lanes; six of the
//    fifteen per pass are read, the others are products of two of those
//    (pass_twiddles), which halves the kernel's L1 traffic for twiddles at
//    the cost of about one float ulp in nine of them; the one-pair kernels
//    form theirs the same way, so the outputs stay bit-identical.
// Scope: n = 4096, MODE_PEAKS, the whole lag window with bins a multiple of
// 32 lags and at most KEYCAP bins (the benchmark's and the refine's layout);
// the launcher sends every other run to flat_kernel / rows_kernel.
#pragma once
#include <cstdint>
#include "packed_passes.cuh"

namespace mfb {

struct Flat2Geo {
  static constexpr int N = 4096;
  static constexpr int T = 256;                 // threads per pair slot
  static constexpr int BUF = N + N / 16;        // padded float4 records
  static constexpr int KEYS = 2 * 2 * KEYCAP;   // two pairs, double-buffered
  static constexpr int SMEM = BUF * 16 + KEYS * 8;
  static constexpr int TW = 15 * 16 + 15 * 256; // float4 twiddles of passes 1 and 2
};

// Items [ibeg, iend) of a launch: item i = pairs 2i, 2i+1 of the dense block
// (row = d*nt + t) or of the row list.  a.twid points at Flat2Geo::TW float4
// records: pass 1 at (q-1)*16 + k, pass 2 at 240 + (q-1)*256 + k.
template <int MODE>
__global__ void __launch_bounds__(256, 2)
flat2_kernel(const FlatArgs a) {
  static_assert(MODE == MODE_PEAKS, "peaks only");
  using Geo = Flat2Geo;
  constexpr int T = Geo::T;
  extern __shared__ __align__(16) float4 smem4[];
  float4 *buf = smem4;
  unsigned long long *kslots = reinterpret_cast<unsigned long long *>(smem4 + Geo::BUF);
  const float4 *tw4 = reinterpret_cast<const float4 *>(a.twid);

  const int t = threadIdx.x;
  const int lane = t & 31;
  const long long total = a.list ? (long long)(*a.list_count) : (long long)a.nd * a.nt;
  if (a.list && a.trig_total && blockIdx.x == 0 && threadIdx.x == 0)
    *a.trig_total += (unsigned long long)total;
  const long long items = (total + 1) / 2;
  const long long per = items / gridDim.x, extra = items % gridDim.x;
  const long long ibeg = blockIdx.x * per + (blockIdx.x < extra ? blockIdx.x : extra);
  const long long iend = ibeg + per + (blockIdx.x < extra ? 1 : 0);

  const int bs = a.binsize;
  const float inv_bs = 1.0f / (float)bs;
  const int nb = a.nb;
  const unsigned linv = 31u - (unsigned)lane;
  for (int b = t; b < Geo::KEYS; b += T) kslots[b] = 0ull;
  __syncthreads();

  for (long long item = ibeg; item < iend; ++item) {
    const long long pa = 2 * item, pb = 2 * item + 1;
    const bool live_b = pb < total;
    int row_a = a.list ? a.list[pa] : (int)pa;
    int row_b = live_b ? (a.list ? a.list[pb] : (int)pb) : row_a;
    const int da = row_a / a.nt, ta = row_a - da * a.nt;
    const int db = row_b / a.nt, tb = row_b - db * a.nt;
    // ---- pass 0: loads, conjugate products (scalar, into the two lanes) ------
    float2 X[16], Y[16];
    {
      const float2 *ha = a.tmpl + (long long)(a.t0 + ta) * a.tmpl_stride + t;
      const float2 *hb = a.tmpl + (long long)(a.t0 + tb) * a.tmpl_stride + t;
      const float2 *dpa = a.data + (long long)(a.d0 + da) * a.data_stride + t;
      const float2 *dpb = a.data + (long long)(a.d0 + db) * a.data_stride + t;
      if (da == db) {
#pragma unroll
        for (int s = 0; s < 16; s++) {
          const float2 d = __ldg(dpa + T * s);
          const float2 h = __ldg(ha + T * s), g = __ldg(hb + T * s);
          X[s].x = fmaf(d.x, h.x, d.y * h.y);
          Y[s].x = fmaf(d.y, h.x, -d.x * h.y);
          X[s].y = fmaf(d.x, g.x, d.y * g.y);
          Y[s].y = fmaf(d.y, g.x, -d.x * g.y);
        }
      } else {
#pragma unroll
        for (int s = 0; s < 16; s++) {
          const float2 d = __ldg(dpa + T * s), e = __ldg(dpb + T * s);
          const float2 h = __ldg(ha + T * s), g = __ldg(hb + T * s);
          X[s].x = fmaf(d.x, h.x, d.y * h.y);
          Y[s].x = fmaf(d.y, h.x, -d.x * h.y);
          X[s].y = fmaf(e.x, g.x, e.y * g.y);
          Y[s].y = fmaf(e.y, g.x, -e.x * g.y);
        }
      }
    }
    p2::dft16(X, Y);
    __syncthreads();           // the previous item's parks and keys are read
    {
      float4 *p0 = buf + pad16(t * 16);
#pragma unroll
      for (int q = 0; q < 16; q++) p0[q] = make_float4(X[q].x, X[q].y, Y[q].x, Y[q].y);
    }
    __syncthreads();
    // ---- pass 1 (span 16) ------------------------------------------------------
    {
      const float4 *pl = buf + pad16(t);
#pragma unroll
      for (int q = 0; q < 16; q++) {
        const float4 r = pl[q * (T + T / 16)];
        X[q] = make_float2(r.x, r.y);
        Y[q] = make_float2(r.z, r.w);
      }
      const int k = t & 15;
      p2::pass_twiddles(X, Y, tw4 + k, 16);
      p2::dft16(X, Y);
      __syncthreads();
      float4 *ps = buf + pad16((t >> 4) * 256 + k);
#pragma unroll
      for (int q = 0; q < 16; q++) ps[q * 17] = make_float4(X[q].x, X[q].y, Y[q].x, Y[q].y);
      __syncthreads();
    }
    // ---- pass 2 (span 256) -----------------------------------------------------
    {
      const float4 *pl = buf + pad16(t);
#pragma unroll
      for (int q = 0; q < 16; q++) {
        const float4 r = pl[q * (T + T / 16)];
        X[q] = make_float2(r.x, r.y);
        Y[q] = make_float2(r.z, r.w);
      }
      p2::pass_twiddles(X, Y, tw4 + 240 + t, 256);
      p2::dft16(X, Y);
      __syncthreads();         // buf is free: parks go there
    }
    // Thread t holds z[t + 256 q] of pair A in lane x, of pair B in lane y.
    // ---- per-bin argmax: one redux per slot, warp and pair ---------------------
    unsigned long long *keys = kslots + (int)(item & 1) * 2 * KEYCAP;   // [2][KEYCAP]
    {
      float2 *park = reinterpret_cast<float2 *>(buf);
      // lane q keeps pair A's slot-q maximum, lane 16 + q pair B's
      unsigned my = 0u;
#pragma unroll
      for (int q = 0; q < 16; q++) {
        const float2 m2 = p2::fma(X[q], X[q], p2::mul(Y[q], Y[q]));
        const unsigned ka = (m2.x > a.t2) ? ((__float_as_uint(m2.x) & ~31u) | linv) : 0u;
        const unsigned kb = (live_b && m2.y > a.t2) ? ((__float_as_uint(m2.y) & ~31u) | linv) : 0u;
        const unsigned xa = __reduce_max_sync(0xffffffffu, ka);
        const unsigned xb = __reduce_max_sync(0xffffffffu, kb);
        const int at = 2 * pad16(t + T * q);
        if (ka != 0u && ka == xa) park[at] = make_float2(X[q].x, Y[q].x);
        if (kb != 0u && kb == xb) park[at + 1] = make_float2(X[q].y, Y[q].y);
        my = ((lane & 15) == q) ? (lane < 16 ? xa : xb) : my;
      }
      if (my != 0u) {
        const int q = lane & 15;
        const int k = ((t & ~31) | (31 - (int)(my & 31u))) + T * q;
        const int bin = bin_of((t & ~31) + T * q, bs, inv_bs);
        atomicMax(keys + (lane >> 4) * KEYCAP + bin,
                  ((unsigned long long)(my & ~31u) << 32) | (unsigned)(~k));
      }
    }
    __syncthreads();
    // ---- outputs: threads [0, nb) pair A, [128, 128 + nb) pair B ----------------
    {
      const int sel = t >> 7, b = t & 127;
      const bool mine = b < nb && (sel == 0 || live_b);
      if (mine) {
        const unsigned long long kk = keys[sel * KEYCAP + b];
        const long long row = sel ? row_b : row_a;
        long long ix = -1;
        float2 val = make_float2(0.f, 0.f);
        if (kk != 0ull) {
          const int k = (int)(~(unsigned)kk);
          ix = k;
          val = reinterpret_cast<const float2 *>(buf)[2 * pad16(k) + sel];
        }
        const long long o = row * nb + b;
        a.out_idx[o * a.rs] = ix;
        a.out_val[o * a.rs] = val;
        if (a.host_rec)   // 16-byte store over the host link into the host table
          a.host_rec[o] = make_int4((int)(unsigned)(unsigned long long)ix,
                                    (int)(unsigned)((unsigned long long)ix >> 32),
                                    __float_as_int(val.x), __float_as_int(val.y));
        if (a.out_cnt && kk != 0ull) atomicAdd(a.out_cnt + row, 1);
      }
      // clear the other parity's keys for the next item (not read before the
      // next item's first barrier)
      unsigned long long *nxt = kslots + (int)((item + 1) & 1) * 2 * KEYCAP;
      if (b < nb && (sel == 0 || live_b)) nxt[sel * KEYCAP + b] = 0ull;
    }
  }
}

// The same pair transform for bins and windows in whole multiples of 256 lags
// (n/16 and up: the usual bank run), with the threads of passes 1 and 2
// numbered so that the second exchange stays inside half-warps.  Digits: point
// f = n0 + 16 n1 + 256 n2, lag k = K0 + 16 K1 + 256 K2.
//   pass 0  thread n0 + 16 n1 transforms over n2 (coalesced loads)
//   pass 1  thread n0 + 16 K0 transforms over n1: CTA-wide exchange
//   pass 2  thread K1 + 16 K0 transforms over n0: exchanged among the 16 threads
//           of K0, in their own region of the buffer
// A warp (two K0, all K1) ends with 32 lags of every block of 256, so with bins
// of whole blocks a slot's warp maximum is one redux; the winner's value goes
// to a small stage instead of the exchange buffer, and an item's outputs are
// written between the next item's two barriers.  Two CTA barriers per item
// instead of six, so warps drift apart and one's FP32 work covers another's
// shared-memory traffic: 204 -> 184 us for 16 x 1024 pairs, binsize 256, on a B200
// (43% FMA pipe, 53% L1; 16 warps per SM, so latency, not a pipe, is the bound).
// Same operations and key order as flat2_kernel: the outputs are bit-identical.
// Bins of other sizes stay with flat2_kernel: their warps' 32 lags, spread over 256,
// would lie in several bins and need a reduction each.
struct Flat2wGeo {
  static constexpr int N = 4096, T = 256;
  static constexpr int REGION = 16 * 17;               // float4 records per K0 (rows of 17: conflict-free)
  static constexpr int BUF = 16 * REGION;
  static constexpr int NB = N / 256;                   // at most 16 bins
  static constexpr int STAGE = 2 * 8 * 16 * 2;         // float2: parity, warp, slot, pair
  static constexpr int SMEM = BUF * 16 + STAGE * 8 + 2 * 2 * NB * 8;
  static constexpr int TW = Flat2Geo::TW;              // pass 2 entries in thread order
};

__global__ void __launch_bounds__(256, 2) flat2w_kernel(const FlatArgs a) {
  using Geo = Flat2wGeo;
  constexpr int T = Geo::T, NB = Geo::NB;
  extern __shared__ __align__(16) float4 smem4[];
  float4 *buf = smem4;
  float2 *stage = reinterpret_cast<float2 *>(smem4 + Geo::BUF);                     // [2][8][16][2]
  unsigned long long *kslots = reinterpret_cast<unsigned long long *>(stage + Geo::STAGE);   // [2][2][NB]
  const float4 *tw4 = reinterpret_cast<const float4 *>(a.twid);

  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int lo = t & 15, hi = t >> 4;
  const long long total = a.list ? (long long)(*a.list_count) : (long long)a.nd * a.nt;
  if (a.list && a.trig_total && blockIdx.x == 0 && threadIdx.x == 0)
    *a.trig_total += (unsigned long long)total;
  const long long items = (total + 1) / 2;
  const long long per = items / gridDim.x, extra = items % gridDim.x;
  const long long ibeg = blockIdx.x * per + (blockIdx.x < extra ? blockIdx.x : extra);
  const long long iend = ibeg + per + (blockIdx.x < extra ? 1 : 0);
  const int nb = a.nb;
  const int q0 = a.ws >> 8, q1 = a.we >> 8, bsq = a.binsize >> 8;   // window and bins in blocks of 256
  // rank of this lane's lag K0 + 16 K1 among the warp's
  const unsigned linv = 31u - (unsigned)(2 * lo + (lane >> 4));
  if (t < 2 * 2 * NB) kslots[t] = 0ull;

  int prev_a = 0, prev_b = -1;
  // Outputs of the item whose keys have parity par: threads [0, nb) pair A,
  // [128, 128 + nb) pair B; keys are cleared for the item two on.
  auto outputs = [&](int par) {
    const int sel = t >> 7, b = t & 127;
    if (b < nb && (sel == 0 || prev_b >= 0)) {
      unsigned long long *key = kslots + (par * 2 + sel) * NB + b;
      const unsigned long long kk = *key;
      long long ix = -1;
      float2 val = make_float2(0.f, 0.f);
      if (kk != 0ull) {
        *key = 0ull;
        const int k = (int)(~(unsigned)kk);
        ix = k;
        val = stage[((par * 8 + ((k & 15) >> 1)) * 16 + (k >> 8)) * 2 + sel];
      }
      const long long row = sel ? prev_b : prev_a;
      const long long o = row * nb + b;
      a.out_idx[o * a.rs] = ix;
      a.out_val[o * a.rs] = val;
      if (a.host_rec)   // 16-byte store over the host link into the host table
        a.host_rec[o] = make_int4((int)(unsigned)(unsigned long long)ix,
                                  (int)(unsigned)((unsigned long long)ix >> 32),
                                  __float_as_int(val.x), __float_as_int(val.y));
      if (a.out_cnt && kk != 0ull) atomicAdd(a.out_cnt + row, 1);
    }
  };

  for (long long item = ibeg; item < iend; ++item) {
    const int par = (int)(item & 1);
    const long long pa = 2 * item, pb = 2 * item + 1;
    const bool live_b = pb < total;
    const int row_a = a.list ? a.list[pa] : (int)pa;
    const int row_b = live_b ? (a.list ? a.list[pb] : (int)pb) : row_a;
    const int da = row_a / a.nt, ta = row_a - da * a.nt;
    const int db = row_b / a.nt, tb = row_b - db * a.nt;
    // ---- pass 0: loads, conjugate products (scalar, into the two lanes) ------
    float2 X[16], Y[16];
    {
      const float2 *ha = a.tmpl + (long long)(a.t0 + ta) * a.tmpl_stride + t;
      const float2 *hb = a.tmpl + (long long)(a.t0 + tb) * a.tmpl_stride + t;
      const float2 *dpa = a.data + (long long)(a.d0 + da) * a.data_stride + t;
      const float2 *dpb = a.data + (long long)(a.d0 + db) * a.data_stride + t;
      if (da == db) {
#pragma unroll
        for (int s = 0; s < 16; s++) {
          const float2 d = __ldg(dpa + T * s);
          const float2 h = __ldg(ha + T * s), g = __ldg(hb + T * s);
          X[s].x = fmaf(d.x, h.x, d.y * h.y);
          Y[s].x = fmaf(d.y, h.x, -d.x * h.y);
          X[s].y = fmaf(d.x, g.x, d.y * g.y);
          Y[s].y = fmaf(d.y, g.x, -d.x * g.y);
        }
      } else {
#pragma unroll
        for (int s = 0; s < 16; s++) {
          const float2 d = __ldg(dpa + T * s), e = __ldg(dpb + T * s);
          const float2 h = __ldg(ha + T * s), g = __ldg(hb + T * s);
          X[s].x = fmaf(d.x, h.x, d.y * h.y);
          Y[s].x = fmaf(d.y, h.x, -d.x * h.y);
          X[s].y = fmaf(e.x, g.x, e.y * g.y);
          Y[s].y = fmaf(e.y, g.x, -e.x * g.y);
        }
      }
    }
    p2::dft16(X, Y);
    __syncthreads();           // the previous item's exchange is read, its keys are final
    {
      float4 *ps = buf + hi * 17 + lo;                 // (K0, n1 = hi, n0 = lo)
#pragma unroll
      for (int q = 0; q < 16; q++)
        ps[q * Geo::REGION] = make_float4(X[q].x, X[q].y, Y[q].x, Y[q].y);
    }
    if (item > ibeg) outputs(par ^ 1);
    __syncthreads();
    // ---- pass 1: thread (n0 = lo, K0 = hi) --------------------------------------
    float4 *mine = buf + hi * Geo::REGION;
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const float4 r = mine[q * 17 + lo];
      X[q] = make_float2(r.x, r.y);
      Y[q] = make_float2(r.z, r.w);
    }
    p2::pass_twiddles(X, Y, tw4 + hi, 16);
    p2::dft16(X, Y);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 16; q++) mine[q * 17 + lo] = make_float4(X[q].x, X[q].y, Y[q].x, Y[q].y);
    __syncwarp();
    // ---- pass 2: thread (K1 = lo, K0 = hi) --------------------------------------
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const float4 r = mine[lo * 17 + q];
      X[q] = make_float2(r.x, r.y);
      Y[q] = make_float2(r.z, r.w);
    }
    p2::pass_twiddles(X, Y, tw4 + 240 + t, 256);
    p2::dft16(X, Y);
    // ---- per-bin argmax: z[hi + 16 lo + 256 q] of pair A in lane x, B in lane y ----
    float mxa = 0.f, mxb = 0.f;
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const float2 m2 = p2::fma(X[q], X[q], p2::mul(Y[q], Y[q]));
      mxa = fmaxf(mxa, m2.x);
      mxb = fmaxf(mxb, m2.y);
    }
    if (__any_sync(0xffffffffu, mxa > a.t2 || (live_b && mxb > a.t2))) {
      float2 *st = stage + (par * 8 + warp) * 32;
      unsigned my = 0u;   // lane q keeps pair A's slot-q maximum, lane 16 + q pair B's
#pragma unroll
      for (int q = 0; q < 16; q++) {
        const float2 m2 = p2::fma(X[q], X[q], p2::mul(Y[q], Y[q]));
        const unsigned ka = (m2.x > a.t2) ? ((__float_as_uint(m2.x) & ~31u) | linv) : 0u;
        const unsigned kb = (live_b && m2.y > a.t2) ? ((__float_as_uint(m2.y) & ~31u) | linv) : 0u;
        const unsigned xa = __reduce_max_sync(0xffffffffu, ka);
        const unsigned xb = __reduce_max_sync(0xffffffffu, kb);
        if (ka != 0u && ka == xa) st[2 * q] = make_float2(X[q].x, Y[q].x);
        if (kb != 0u && kb == xb) st[2 * q + 1] = make_float2(X[q].y, Y[q].y);
        my = (lo == q) ? (lane < 16 ? xa : xb) : my;
      }
      if (my != 0u && lo >= q0 && lo < q1) {
        const int rank = 31 - (int)(my & 31u);
        const int k = 2 * warp + (rank & 1) + 16 * (rank >> 1) + 256 * lo;
        atomicMax(kslots + (par * 2 + (lane >> 4)) * NB + (lo - q0) / bsq,
                  ((unsigned long long)(my & ~31u) << 32) | (unsigned)(~k));
      }
    }
    prev_a = row_a;
    prev_b = live_b ? row_b : -1;
  }
  if (ibeg < iend) {
    __syncthreads();
    outputs((int)((iend - 1) & 1));
  }
}

}  // namespace mfb
