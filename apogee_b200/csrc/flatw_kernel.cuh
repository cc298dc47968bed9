// Fused matched filter at n = 512 ... 16384 for bins and windows in whole blocks
// of n/16 lags (the usual bank run), and the coarse gate at those lengths.
//
// Same pair transform as flat_kernel (same operations in the same order, so the
// outputs are bit-identical); what differs is which thread holds what.  There every
// pass meets at two CTA barriers, so a CTA's warps run its FP32 phases and
// its shared-memory phases together and neither pipe is busy for long.  Here the
// threads of the later passes are numbered so that one exchange stays within
// half-warps, and a pair's outputs are written between the next pair's barriers.
// Digits, with R = R0 (2 ... 16) the first radix and T = n/16 threads per pair:
//
//   n = 256 R:  f = n0 + 16 n1 + 256 n2,  k = K0 + R K1 + T K2
//     pass 0  thread t transforms over n2 (coalesced loads), 16/R butterflies
//     pass 1  thread n0 + 16 K0, over n1: exchanged among the pair's threads
//     pass 2  thread K1 + 16 K0, over n0: exchanged among the 16 threads of K0
//   n = 4096 R:  f = n0 + 16 n1 + 256 n2 + 4096 n3,  k = K0 + R K1 + 16 R K2 + T K3
//     pass 1  thread n1 + 16 n0 + 256 K0, over n2: exchanged among the pair's threads
//     pass 2  thread K1 + 16 n0 + 256 K0, over n1: among the 16 threads of (n0, K0)
//     pass 3  thread K2 + 16 K1 + 256 K0, over n0: among the 256 threads of K0
//
// Every exchange is free of bank conflicts (strides of 17 and 273 float2).  A pair
// slot synchronises by itself (warp, named barrier or CTA barrier), so the slots
// of a CTA drift apart, and 64 registers a thread leave 32 warps per SM.  A warp's
// 32 lags of a block lie in one bin: one redux per block, the winner's value to a
// small stage.
//
// A slot takes every slots-th pair: the rows whose pairs have candidates (a loud data
// row) are then shared by all SMs, and the slots of an SM are on the same data row.
// With a contiguous range per slot the SMs were active 93% (n = 4096) and 79% (16384) of
// the slowest one's time.
//
// Measured on a B200 (us, 16 warps' packed two-pair kernel or flat_kernel before ->
// contiguous ranges -> now): 16 x 1024 pairs at n = 4096, threshold 5.5
// 204 -> 166 -> 159; 6 x 300 at n = 16384 149 -> 118 -> 100.
#pragma once
#include "flat_kernel.cuh"

namespace mfb {

template <int N>
struct FlatWGeo {
  using Geo = FlatGeo<N>;
  static_assert(N >= 512 && N <= 16384, "a pair has at least one warp");
  static constexpr int T = Geo::T, R = Geo::R0, CTA = Geo::CTA, G = Geo::G, PASSES = Geo::PASSES;
  static constexpr int REGION = PASSES == 3 ? 272 : 16 * 273;   // float2 per K0
  static constexpr int BUF = R * REGION;
  static constexpr int WARPS = T / 32;
  static constexpr int STAGE = 2 * WARPS * 16;                  // float2: parity, warp, block
  static constexpr int SLOT = BUF * 8 + STAGE * 8 + 2 * 16 * 8 + 16;   // bytes per pair slot (keys, gate words)
  static constexpr int SMEM = G * SLOT;
  static constexpr int MINB = CTA <= 256 ? 4 : CTA <= 512 ? 2 : 1;
  // twiddles in thread order: pass 1 [q][K0]; n = 4096 R: pass 2 [q][16 K0 + K1]; last pass [q][t]
  static constexpr int OFF2 = 15 * R;
  static constexpr int OFF3 = PASSES == 3 ? OFF2 : OFF2 + 15 * 16 * R;
  static constexpr int TW = OFF3 + 15 * T;
  static_assert(SLOT % 16 == 0, "slots keep 16-byte alignment");
};

template <int N, int MODE>
__global__ void __launch_bounds__(FlatWGeo<N>::CTA, FlatWGeo<N>::MINB) flatw_kernel(const FlatArgs a) {
  using Geo = FlatWGeo<N>;
  constexpr int T = Geo::T, R = Geo::R, G = Geo::G, PASSES = Geo::PASSES, B0 = 16 / R;
  extern __shared__ __align__(16) unsigned char flatw_smem[];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  float2 *buf = reinterpret_cast<float2 *>(flatw_smem + g * Geo::SLOT);
  float2 *stage = buf + Geo::BUF;                                                            // [2][WARPS][16]
  unsigned long long *kslots = reinterpret_cast<unsigned long long *>(stage + Geo::STAGE);   // [2][16]
  unsigned *gslots = reinterpret_cast<unsigned *>(kslots + 2 * 16);                            // [2]
  const int lane = t & 31, warp = t >> 5, lo = t & 15, hi = t >> 4;
  auto sync = [&]() {
    if constexpr (T <= 32) __syncwarp();
    else if constexpr (G == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" :: "r"(1 + g), "n"(T) : "memory");
  };
  const long long total = a.list ? (long long)(*a.list_count) : (long long)a.nd * a.nt;
  if (a.list && a.trig_total && blockIdx.x == 0 && threadIdx.x == 0)
    *a.trig_total += (unsigned long long)total;
  // every slots-th pair (see above)
  const long long slots = (long long)gridDim.x * G, me = (long long)blockIdx.x * G + g;
  const int nb = a.nb;
  const int q0 = a.ws / T, q1 = a.we / T;                       // window and bins in blocks (MODE_PEAKS)
  const int bsq = MODE == MODE_PEAKS ? a.binsize / T : 1;
  // rank of this lane's lag among the warp's: lo first, then the half-warp
  const unsigned linv = 31u - (unsigned)(2 * lo + (lane >> 4));
  if (t < 2 * 16) kslots[t] = 0ull;
  if (t < 2) gslots[t] = 0u;
  sync();

  int prev = 0, par = 1;
  // Outputs of pair `prev`, whose keys have parity par (keys are cleared for the pair two on).
  auto outputs = [&](int par) {
    if constexpr (MODE == MODE_PEAKS) {
      if (t < nb) {
        unsigned long long *key = kslots + par * 16 + t;
        const unsigned long long kk = *key;
        long long ix = -1;
        float2 val = make_float2(0.f, 0.f);
        if (kk != 0ull) {
          *key = 0ull;
          const int k = (int)(~(unsigned)kk), r = k % T;
          const int w = PASSES == 3 ? (r % R) >> 1 : (r % R) * 8 + (((r / R) & 15) >> 1);
          ix = k;
          val = stage[(par * Geo::WARPS + w) * 16 + k / T];
        }
        const long long o = (long long)prev * nb + t;
        a.out_idx[o * a.rs] = ix;
        a.out_val[o * a.rs] = val;
        if (a.host_rec) store_host(a.host_rec, o, ix, val);
        if (a.out_cnt && kk != 0ull) atomicAdd(a.out_cnt + prev, 1);
      }
    } else {
      const unsigned bits = gslots[par];
      const float m = sqrtf(__uint_as_float(bits));
      if (a.coarse_out) {
        if (t == 0) a.coarse_out[prev] = m;
      } else if (bits != 0u && m >= a.gate) {
        if (t == 0) a.fire_list[atomicAdd(a.fire_count, 1)] = prev;
      } else {
        const long long obase = (long long)prev * a.full_nb;
        for (int b = t; b < a.full_nb; b += T) {
          a.out_idx[(obase + b) * a.rs] = -1;
          a.out_val[(obase + b) * a.rs] = make_float2(0.f, 0.f);
        }
      }
    }
  };

  for (long long item = me; item < total; item += slots) {
    par ^= 1;
    const int row = a.list ? a.list[item] : (int)item;
    const int d = row / a.nt, tt = row - d * a.nt;
    cf v[16];
    // ---- pass 0: loads, conjugate product, radix R -----------------------------------
    {
      const float2 *hp = a.tmpl + (long long)(a.t0 + tt) * a.tmpl_stride + t;
      const float2 *dp = a.data + (long long)(a.d0 + d) * a.data_stride + t;
#pragma unroll
      for (int s = 0; s < 16; s++) {
        const float2 x = __ldg(dp + T * s), h = __ldg(hp + T * s);
        v[s].x = fmaf(x.x, h.x, x.y * h.y);
        v[s].y = fmaf(x.y, h.x, -x.x * h.y);
      }
    }
    first_pass<R>(v);
    sync();                    // the previous pair's exchange is read, its keys are final
#pragma unroll
    for (int b = 0; b < B0; b++)
#pragma unroll
      for (int q = 0; q < R; q++) {
        // point j = t + T b of the remaining digits, K0 = q
        constexpr int JB = T / 16;            // n1 + 16 n2 advances by JB per b
        const int at = PASSES == 3 ? q * Geo::REGION + (hi + JB * b) * 17 + lo
                                   : q * Geo::REGION + ((hi >> 4) + R * b) * 273 + (hi & 15) * 17 + lo;
        buf[at] = make_float2(v[b + B0 * q].x, v[b + B0 * q].y);
      }
    if (item != me) outputs(par ^ 1);
    sync();
    if (MODE == MODE_GATE && t == 0) gslots[par ^ 1] = 0u;   // read above; next written a barrier on
    if constexpr (PASSES == 3) {
      float2 *mine = buf + hi * Geo::REGION;
      // ---- pass 1: thread (n0 = lo, K0 = hi) ---------------------------------------
#pragma unroll
      for (int q = 0; q < 16; q++) { const float2 r = mine[q * 17 + lo]; v[q] = {r.x, r.y}; }
      pass_twiddles(v, a.twid + hi, R);
      dft16(v);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 16; q++) mine[q * 17 + lo] = make_float2(v[q].x, v[q].y);
      __syncwarp();
      // ---- pass 2: thread (K1 = lo, K0 = hi) ---------------------------------------
#pragma unroll
      for (int q = 0; q < 16; q++) { const float2 r = mine[lo * 17 + q]; v[q] = {r.x, r.y}; }
    } else {
      const int K0 = t >> 8, mid = hi & 15;
      float2 *reg = buf + K0 * Geo::REGION;
      // ---- pass 1: thread (n1 = lo, n0 = mid, K0) -------------------------------------
      {
        float2 *mine = reg + lo * 17 + mid;
#pragma unroll
        for (int q = 0; q < 16; q++) { const float2 r = mine[q * 273]; v[q] = {r.x, r.y}; }
        pass_twiddles(v, a.twid + K0, R);
        dft16(v);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 16; q++) mine[q * 273] = make_float2(v[q].x, v[q].y);
        __syncwarp();
      }
      // ---- pass 2: thread (K1 = lo, n0 = mid, K0) -------------------------------------
      {
        const float2 *mine = reg + lo * 273 + mid;
#pragma unroll
        for (int q = 0; q < 16; q++) { const float2 r = mine[q * 17]; v[q] = {r.x, r.y}; }
        pass_twiddles(v, a.twid + Geo::OFF2 + 16 * K0 + lo, 16 * R);
        dft16(v);
        asm volatile("bar.sync %0, 256;" :: "r"(1 + K0) : "memory");   // the threads of K0 have read
#pragma unroll
        for (int q = 0; q < 16; q++) reg[mid * 273 + lo * 17 + q] = make_float2(v[q].x, v[q].y);
        asm volatile("bar.sync %0, 256;" :: "r"(1 + K0) : "memory");
      }
      // ---- pass 3: thread (K2 = lo, K1 = mid, K0) -------------------------------------
      const float2 *mine = reg + mid * 17 + lo;
#pragma unroll
      for (int q = 0; q < 16; q++) { const float2 r = mine[q * 273]; v[q] = {r.x, r.y}; }
    }
    pass_twiddles(v, a.twid + Geo::OFF3 + t, T);
    dft16(v);
    // ---- z of block q, this thread's lag in it, in v[q] -----------------------------------
    if constexpr (MODE == MODE_PEAKS) {
      if (any_candidate(v, a.t2, true, 0xffffffffu)) {
        float2 *st = stage + (par * Geo::WARPS + warp) * 16;
        unsigned my = 0u;      // lane q keeps block q's maximum
#pragma unroll
        for (int q = 0; q < 16; q++) {
          const float m2 = fmaf(v[q].x, v[q].x, v[q].y * v[q].y);
          const unsigned key = (m2 > a.t2) ? ((__float_as_uint(m2) & ~31u) | linv) : 0u;
          const unsigned mx = __reduce_max_sync(0xffffffffu, key);
          if (key != 0u && key == mx) st[q] = make_float2(v[q].x, v[q].y);
          my = (lane == q) ? mx : my;
        }
        if (my != 0u && lane >= q0 && lane < q1) {
          const int rank = 31 - (int)(my & 31u), half = rank & 1, dig = rank >> 1;
          const int in = PASSES == 3 ? 2 * warp + half + R * dig
                                     : (warp >> 3) + R * (2 * (warp & 7) + half) + 16 * R * dig;
          atomicMax(kslots + par * 16 + (lane - q0) / bsq,
                    ((unsigned long long)(my & ~31u) << 32) | (unsigned)(~(in + T * lane)));
        }
      }
    } else {
      float best = 0.f;
      if (a.ws == 0 && a.we == N) {
#pragma unroll
        for (int q = 0; q < 16; q++) best = fmaxf(best, fmaf(v[q].x, v[q].x, v[q].y * v[q].y));
      } else {
        const int in = PASSES == 3 ? hi + R * lo : (t >> 8) + R * ((hi & 15) + 16 * lo);
#pragma unroll
        for (int q = 0; q < 16; q++) {
          const int k = in + T * q;
          if (k >= a.ws && k < a.we) best = fmaxf(best, fmaf(v[q].x, v[q].x, v[q].y * v[q].y));
        }
      }
      const unsigned mx = __reduce_max_sync(0xffffffffu, best > a.t2 ? __float_as_uint(best) & ~31u : 0u);
      if (lane == 0 && mx != 0u) atomicMax(gslots + par, mx);
    }
    prev = row;
  }
  if (me < total) {
    sync();
    outputs(par);
  }
}

}  // namespace mfb
