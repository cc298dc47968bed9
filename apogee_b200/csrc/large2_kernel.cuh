// Fused matched filter for n = 32768 ... 1048576 in one persistent launch: the
// four-step split of large_kernel.cuh, two pairs per thread in packed FP32x2.
//
// With n = N1 * N2, f = f1 + N1 f2 and k = N2 k1 + k2, an item (pairs 2i and
// 2i+1 of the dense block, template-major, or of the row list) takes
//   N1/C units of kind A   C adjacent columns f1: product, N2-point transform over
//                          f2, twiddle W_n^(f1 k2), store Y[k2][f1];
//   N2/G units of kind B   G adjacent rows k2: N1-point transform over f1, per-bin
//                          maxima, merged across CTAs into 16-byte records;
// of 4096 points per pair each (256 threads of 16 points).  Both transforms
// exchange float4 records (re_A, re_B, im_A, im_B) through 64 KB of shared memory,
// so two CTAs fit on an SM.
//
// Why one launch: as separate launches per L2-sized batch (A, B, finalize and a
// memset), a launch's last wave and the gaps left the SMs active 82% (A) and
// 66% (B) of the time at n = 65536, and both passes were issue bound while
// active (62% and 73%), which the packed arithmetic halves.
//
// Tickets of one counter are handed out in the order A(0) ... A(D-1), then A(i)
// and B(i-D) for i = D ..., then the last D items' B; a ticket is `grp`
// neighbouring units of one item.  Items go through a ring of scratch slots.
// B(i) waits until A(i) is complete, A(i) until the item that had its slot
// before is finalized: always work of smaller tickets.  The CTA that completes an
// item's last B ticket finalizes it (records -> outputs) before its next
// ticket but one, and before it waits for anything.  A CTA holds at most its
// current ticket and the next one it has drawn, so the smallest unfinished ticket
// is being worked on and never waits -- whatever CTAs are resident.  D and the ring
// put at least two tickets per CTA between an item's last A ticket and its first B
// ticket, and again until its slot is wanted, so in steady state nothing waits,
// and both kinds of unit run side by side.  Waits are bounded (LARGE2_SPIN looks); a wait
// that runs out sets the plan's error word and every CTA stops taking tickets.
// The last CTA to leave resets the counters, and the records of a launch that gave up; a
// finalized item leaves its records zero.  So no launch spoils a later one as long as
// launches on the same counters follow one another (see run_large, mfb_api.cu).
//
// What a unit costs beside its arithmetic is latency: a ticket is drawn one ahead;
// thread 0 decodes it and looks at its dependency while the current ticket's
// first loads are in flight; completion is one release by thread 0 after the
// ticket's last barrier, which the other warps do not wait for; and the rows of
// a B unit stay within their warps.
// The arithmetic (products, passes, twiddles, key order) is that of the
// one-pair kernels, so the outputs equal the cluster kernel's.
//
// Measured on a B200 against the per-batch launches: n = 65536, 4 x 257 pairs,
// binsize 4096: 512 -> 302 us; n = 262144, 4 x 256: 2400 -> 1525 us.  On the way, at
// n = 65536: one ticket per unit with every wait, fence and decode in line 450 us;
// those off the critical path 383; four units per ticket and batches of 150 items
// (450 MB of scratch) 307; per-item dependencies instead of batches (205 MB) 303, with two
// units per ticket 310 (103 MB), with one 363.  One pair per thread was slower: 64 registers
// and four CTAs per SM 322 (n = 262144: 1803 against 1538), 80 and three 309 (1612).  What bounds it now: latency at 16
// warps per SM (128 registers) -- FMA pipe ~40%, issue ~37%, warps waiting at the exchange
// barrier of A and on loads.
#pragma once
#include "large_kernel.cuh"
#include "packed_passes.cuh"

namespace mfb {

constexpr int LARGE2_GROUP = 4;                // units per ticket, at most
constexpr unsigned LARGE2_SPIN = 1u << 22;
constexpr int LARGE2_BUF = 4096 + 4096 / 16;   // float4 records of the exchange buffer

// Counters, zero between launches; the three arrays of one entry per ring slot
// follow: tickets of kind A and B finished and items finalized in the slot, all
// cumulative over the launch.
struct Large2Ctl {
  unsigned long long ticket;
  unsigned exits;           // CTAs that left, and in the high half those that gave up
  int err;                  // a wait ran out in this launch
};

struct Large2Args {
  LargeArgs a;              // inputs, window, bins and outputs (not its scratch or tables)
  const float4 *tw1, *tw2;  // passes of the N1- and N2-point transforms, (wr, wr, wi, wi)
  const float2 *anchors;    // [N1/C][5][256]: pass A's twiddle at q = 0, 4, 8, 12, and its step
  float4 *Y;                // [ring][n]
  int nkeys, kmod;          // bin keys per pair; kmod > 0: keys by (k1, bin mod kmod), else by bin
  uint4 *rec;               // [ring][2][nb] {re, im, ~lag, |z|^2 bits}, zero between launches
  Large2Ctl *ctl;
  int *err;                 // mapped host word, set when a wait ran out
  int ring;                 // slots
  unsigned spin;            // LARGE2_SPIN
  int hold;                 // tests: added to the count of A tickets that B waits for
};

enum { L2_A = 0, L2_B = 1, L2_END = 2 };

// Keys of a unit of kind B, where bins are not shared by whole warps: a unit sees G
// neighbouring lags of every k1 (aligned to G), so of narrow bins it sees a few per k1
// (`kmod`, a power of two; one where bins and window are multiples of G) and needs
// N1 * kmod keys instead of one per bin.  4096 keys for each of two pairs left one CTA per
// SM and were scanned whole by every unit: 4096 bins, threshold 0, n = 65536, 4 x 128 pairs
// 1557 -> 385 us (the per-batch launches before: 861), n = 262144, 4 x 64 2344 -> 778 (1611).
__host__ __device__ inline void large2_keys(int N1, int G, int bs, int ws, int nb, int &nkeys, int &kmod) {
  int S = bs % G == 0 && ws % G == 0 ? 1 : 2;
  while (S > 1 && S < (G + bs - 2) / bs + 1) S *= 2;
  kmod = (long long)N1 * S < nb ? S : 0;
  nkeys = kmod ? N1 * S : nb;
}

// Items between an item's A and B tickets, for `per` tickets per item and a
// grid of `grid` CTAs: two tickets per CTA and a tenth.
__host__ __device__ inline long long large2_delay(int grid, int per) { return 11LL * grid / (5 * per) + 1; }

// Columns per unit of kind A.
template <int N2>
__host__ __device__ constexpr int large2_cols() { return 256 / (N2 / 16); }

// anchors[tile][j][tid]: W_n^(f1 (t + T2 4 j)) for j < 4, W_n^(f1 T2) for j = 4
// (the values pass_a_twiddle takes from the two-level table).
template <int N2>
__global__ void large2_anchors(const LargeArgs a, float2 *out) {
  constexpr int T2 = N2 / 16, C = large2_cols<N2>();
  const int tile = blockIdx.x, c = threadIdx.x % C, t = threadIdx.x / C, f1 = tile * C + c;
  const unsigned nm = (unsigned)(a.n - 1);
  for (int j = 0; j < 5; j++) {
    const unsigned m = j < 4 ? (unsigned)f1 * (unsigned)(t + T2 * 4 * j) : (unsigned)f1 * (unsigned)T2;
    const cf w = wn_table(a, m & nm);
    out[((long long)tile * 5 + j) * 256 + threadIdx.x] = make_float2(w.x, w.y);
  }
}

__device__ __forceinline__ unsigned ld_acquire32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release32(unsigned *p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(p) : "memory");
}
__device__ __forceinline__ unsigned atom_add_acq_rel32(unsigned *p) {
  unsigned v;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// A decoded ticket: tickets [unit, unit + grp) of its kind and item; ready: what
// it depends on was complete when thread 0 looked; fin: item to finalize before it, or -1.
struct Large2Ticket {
  int kind, unit, ready;
  long long item, fin;
};

template <int N1, int N2>
__global__ void __launch_bounds__(256, 2) large2_kernel(const Large2Args g) {
  constexpr int n = N1 * N2;
  constexpr int T2 = N2 / 16, C = large2_cols<N2>(), UA = N1 / C;
  constexpr int T1 = N1 / 16, G = 256 / T1, UB = N2 / G, ROW = FlatGeo<N1>::BUF;
  static_assert(C * T2 == 256 && G * T1 == 256 && G * ROW <= LARGE2_BUF && N2 * C <= LARGE2_BUF, "");
  extern __shared__ __align__(16) float4 large2_smem[];
  float4 *buf = large2_smem;
  unsigned long long *keys = reinterpret_cast<unsigned long long *>(buf + LARGE2_BUF);   // [2][nkeys]
  __shared__ Large2Ticket s_tk[2];
  __shared__ int s_ok;
  __shared__ long long s_fin;
  __shared__ float2 s_stage[8 * 32];            // per warp: slot winners of pair A, then B
  const LargeArgs &a = g.a;
  const int tid = threadIdx.x, lane = tid & 31;
  const long long total = a.list_count ? (long long)*a.list_count : a.total;
  const long long N = (total + 1) / 2;                   // items
  if (N == 0) return;
  const int nb = a.nb, nb2 = 2 * nb, nk = g.nkeys, ring = g.ring;
  unsigned *a_done = reinterpret_cast<unsigned *>(g.ctl + 1), *b_done = a_done + ring, *f_done = b_done + ring;
  // units per ticket: keep at least four tickets of kind A per CTA
  int grp = LARGE2_GROUP;
  while (grp > 1 && N * UA < 4LL * grp * gridDim.x) grp >>= 1;
  const int gA = UA / grp, gB = UB / grp;               // tickets per item (UA, UB are multiples of 8)
  long long D = large2_delay((int)gridDim.x, gA + gB);
  if (D > N) D = N;
  if (ring < N && D > ring - 1) D = ring - 1;           // A(i) comes after B(i - ring); ring >= 2
  const int bs = a.binsize;
  const float inv_bs = 1.0f / (float)bs;
  unsigned smask = 0u, srank = 0u;
  if (a.seg > 0) bin_segment(T1, a.seg, smask, srank);
  else
    for (int b = tid; b < 2 * nk; b += 256) keys[b] = 0ull;

  // x / d and its remainder, in 32 bits when x allows.
  auto div = [](unsigned long long x, unsigned d, unsigned &r) {
    const unsigned long long q = (x >> 32) ? x / d : (unsigned long long)((unsigned)x / d);
    r = (unsigned)(x - q * d);
    return (long long)q;
  };
  // What a ticket depends on: *ctr >= need.
  auto depends = [&](const Large2Ticket &k, unsigned &need) {
    unsigned slot;
    const unsigned round = (unsigned)div((unsigned long long)k.item, (unsigned)ring, slot);
    need = k.kind == L2_A ? round : (round + 1) * gA + g.hold;
    return (k.kind == L2_A ? f_done : a_done) + slot;
  };
  // thread 0: ticket x into s_tk[i].
  auto take = [&](int i, unsigned long long x, long long fin) {
    Large2Ticket k;
    k.kind = L2_END;
    k.item = 0;
    k.ready = 1;
    k.fin = fin;
    unsigned u = 0;
    if (x < (unsigned long long)D * gA) { k.kind = L2_A; k.item = div(x, gA, u); }
    else {
      x -= (unsigned long long)D * gA;
      const unsigned long long mid = (unsigned long long)(N - D) * (gA + gB);
      if (x < mid) {
        const long long j = div(x, gA + gB, u);
        if (u < (unsigned)gA) { k.kind = L2_A; k.item = D + j; }
        else { k.kind = L2_B; k.item = j; u -= gA; }
      } else {
        x -= mid;
        if (x < (unsigned long long)D * gB) { k.kind = L2_B; k.item = N - D + div(x, gB, u); }
      }
    }
    k.unit = (int)u * grp;
    if (k.kind != L2_END) {
      unsigned need;
      const unsigned *ctr = depends(k, need);
      k.ready = need == 0 || ld_acquire32(ctr) >= need;
    }
    s_tk[i] = k;
  };
  // thread 0: bounded wait for s_tk[i]'s dependency.
  auto wait = [&](int i) {
    unsigned need, spins = 0;
    const unsigned *ctr = depends(s_tk[i], need);
    while (ld_acquire32(ctr) < need) {
      if (++spins > g.spin || *(volatile int *)&g.ctl->err) {
        *(volatile int *)&g.ctl->err = 1;
        *(volatile int *)g.err = 1;
        __threadfence_system();
        return 0;
      }
      __nanosleep(64);
    }
    return 1;
  };
  // All threads: the item's records -> outputs, and its slot is free.
  auto finalize = [&](long long item) {
    const int slot = (int)(item % ring);
    for (int b2 = tid; b2 < nb2; b2 += 256) {
      const int sel = b2 >= nb, b = b2 - sel * nb;
      const long long pi = 2 * item + sel;
      if (pi >= total) continue;
      uint4 *p = g.rec + (long long)slot * nb2 + b2;
      const uint4 r = __ldcg(p);
      int row, d, t;
      large_pair(a, pi, row, d, t);
      const long long o = ((long long)row * nb + b) * a.rs;
      if (r.w == 0u && r.z == 0u) {
        a.out_idx[o] = -1;
        a.out_val[o] = make_float2(0.f, 0.f);
      } else {
        __stcg(p, make_uint4(0u, 0u, 0u, 0u));
        a.out_idx[o] = (long long)(int)(~r.z);
        a.out_val[o] = make_float2(__uint_as_float(r.x), __uint_as_float(r.y));
        if (a.out_cnt) atomicAdd(a.out_cnt + row, 1);
      }
    }
    __syncthreads();
    if (tid == 0) red_release32(f_done + slot);
  };

  // thread 0: the next ticket; the last B ticket's item, and its place in that item's count
  unsigned long long next = 0;
  long long b_item = -1;
  unsigned b_old = 0;
  auto finished = [&]() {      // the item if that ticket completed it, else -1
    if (b_item < 0) return -1LL;
    const long long item = b_item;
    b_item = -1;
    return b_old + 1 == (unsigned)(item / ring + 1) * (unsigned)gB ? item : -1LL;
  };
  if (tid == 0) {
    take(0, atomicAdd(&g.ctl->ticket, 1ull), -1);
    next = atomicAdd(&g.ctl->ticket, 1ull);
  }
  __syncthreads();
  bool gave_up = false;
  for (int par = 0;; par ^= 1) {
    const Large2Ticket tk = s_tk[par];
    if (tk.fin >= 0) finalize(tk.fin);
    if (tk.kind == L2_END || !tk.ready) {
      // nothing may stay pending across a wait or at the end
      if (tid == 0) s_fin = finished();
      __syncthreads();
      if (s_fin >= 0) finalize(s_fin);
      if (tk.kind == L2_END) break;
      if (tid == 0) s_ok = wait(par);
      __syncthreads();
      if (!s_ok) { gave_up = true; break; }
    }
    const int slot = (int)(tk.item % ring);
    if (tk.kind == L2_A) {
      {
        const int tile0 = tk.unit;
        const long long pa = 2 * tk.item, pb = pa + 1;
        const int c = tid % C, t = tid / C;
        int row, da, ta, db, tb;
        large_pair(a, pa, row, da, ta);
        if (pb < total) large_pair(a, pb, row, db, tb);
        else { db = da; tb = ta; }
        const int off = tile0 * C + c + N1 * t;
        const float2 *ha = a.tmpl + (long long)(a.t0 + ta) * n + off;
        const float2 *hb = a.tmpl + (long long)(a.t0 + tb) * n + off;
        const float2 *dpa = a.data + (long long)(a.d0 + da) * n + off;
        const float2 *dpb = a.data + (long long)(a.d0 + db) * n + off;
        const float2 *an = g.anchors + (long long)tile0 * 5 * 256 + tid;
        float4 *yp = g.Y + (long long)slot * n + off;   // [k2 = t + T2 s][f1]
#pragma unroll 1
        for (int i = 0; i < grp; i++) {
          float2 X[16], Y[16];
          if (ta == tb) {
#pragma unroll
            for (int s = 0; s < 16; s++) {
              const int f = N1 * T2 * s;
              const float2 h = __ldg(ha + f), d = __ldg(dpa + f), e = __ldg(dpb + f);
              X[s].x = fmaf(d.x, h.x, d.y * h.y);
              Y[s].x = fmaf(d.y, h.x, -d.x * h.y);
              X[s].y = fmaf(e.x, h.x, e.y * h.y);
              Y[s].y = fmaf(e.y, h.x, -e.x * h.y);
            }
          } else {
#pragma unroll
            for (int s = 0; s < 16; s++) {
              const int f = N1 * T2 * s;
              const float2 h = __ldg(ha + f), k = __ldg(hb + f), d = __ldg(dpa + f), e = __ldg(dpb + f);
              X[s].x = fmaf(d.x, h.x, d.y * h.y);
              Y[s].x = fmaf(d.y, h.x, -d.x * h.y);
              X[s].y = fmaf(e.x, k.x, e.y * k.y);
              Y[s].y = fmaf(e.y, k.x, -e.x * k.y);
            }
          }
          if (i == 0 && tid == 0) take(par ^ 1, next, finished());
          p2::passes<N2, true, false>(X, Y, buf, g.tw2, t, [c](int j) { return j * C + c; },
                                      []() { __syncthreads(); });
          const float2 st = __ldg(an + 4 * 256);
          cf w;
#pragma unroll
          for (int s = 0; s < 16; s++) {
            if ((s & 3) == 0) { const float2 x = __ldg(an + (s >> 2) * 256); w = {x.x, x.y}; }
            else w = cmul(w, cf{st.x, st.y});
            p2::twiddle(X[s], Y[s], make_float4(w.x, w.x, w.y, w.y));
          }
#pragma unroll
          for (int s = 0; s < 16; s++)
            yp[N1 * T2 * s] = make_float4(X[s].x, X[s].y, Y[s].x, Y[s].y);
          ha += C; hb += C; dpa += C; dpb += C; an += 5 * 256; yp += C;
        }
      }
    } else {
      {
        const bool live_b = 2 * tk.item + 1 < total;
        const int gr = tid / T1, t = tid % T1;
        int k2base = tk.unit * G;
        const float4 *yp = g.Y + (long long)slot * n + (long long)(k2base + gr) * N1 + t;
        uint4 *rec = g.rec + (long long)slot * nb2;
        float4 *rbuf = buf + gr * ROW;
#pragma unroll 1
        for (int i = 0; i < grp; i++, k2base += G, yp += G * N1) {
          const int k2 = k2base + gr;
          float2 X[16], Y[16];
#pragma unroll
          for (int s = 0; s < 16; s++) {
            const float4 r = __ldcg(yp + T1 * s);
            X[s] = make_float2(r.x, r.y);
            Y[s] = make_float2(r.z, r.w);
          }
          if (i == 0 && tid == 0) take(par ^ 1, next, finished());
          p2::passes<N1, false, true>(X, Y, rbuf, g.tw1, t, [](int j) { return pad16(j); },
                                      []() { if constexpr (T1 > 32) __syncthreads(); else __syncwarp(); });
          // thread t holds z[N2 k1 + k2], k1 = t + T1 q, of both pairs
          float mxa = 0.f, mxb = 0.f;
#pragma unroll
          for (int s = 0; s < 16; s++) {
            const float2 m2 = p2::fma(X[s], X[s], p2::mul(Y[s], Y[s]));
            mxa = fmaxf(mxa, m2.x);
            mxb = fmaxf(mxb, m2.y);
          }
          const bool any = mxa > a.t2 || (live_b && mxb > a.t2);
          if (a.seg > 0) {
            // every slot of the warp lies in one bin: lane s keeps slot s's best of pair A,
            // lane 16 + s of pair B, and the lanes merge them into the records
            if (__any_sync(0xffffffffu, any)) {
              float2 *stage = s_stage + (tid >> 5) * 32;
              unsigned mk = 0u;
#pragma unroll
              for (int s = 0; s < 16; s++) {
                const int lag = N2 * (t + T1 * s) + k2;
                const float2 m2 = p2::fma(X[s], X[s], p2::mul(Y[s], Y[s]));
                const bool in = lag >= a.ws && lag < a.we;
                const unsigned ka = in && m2.x > a.t2 ? (__float_as_uint(m2.x) & ~31u) | (31u - srank) : 0u;
                const unsigned kb = in && live_b && m2.y > a.t2
                                        ? (__float_as_uint(m2.y) & ~31u) | (31u - srank) : 0u;
                const unsigned xa = __reduce_max_sync(0xffffffffu, ka);
                const unsigned xb = __reduce_max_sync(0xffffffffu, kb);
                if (ka != 0u && ka == xa) stage[s] = make_float2(X[s].x, Y[s].x);
                if (kb != 0u && kb == xb) stage[16 + s] = make_float2(X[s].y, Y[s].y);
                if ((lane & 15) == s) mk = lane < 16 ? xa : xb;
              }
              __syncwarp();
              if (mk != 0u) {
                // the winner's rank is its place in the warp in lag order (t, then row)
                constexpr int R = T1 >= 32 ? 1 : 32 / T1;
                const int rank = 31 - (int)(mk & 31u), s = lane & 15;
                const int tw = T1 >= 32 ? (t & ~31) + rank : rank / R;
                const int rw = T1 >= 32 ? gr : (tid >> 5) * R + rank % R;
                const int lag = N2 * (tw + T1 * s) + k2base + rw;
                const float2 v = stage[lane];
                rec_max(rec + (lane >> 4) * nb + bin_of(lag - a.ws, bs, inv_bs),
                        make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), (unsigned)~lag, mk & ~31u));
              }
            }
          } else if (__syncthreads_or(any)) {
            float2 *park = reinterpret_cast<float2 *>(rbuf);
            if (any) {
#pragma unroll
              for (int s = 0; s < 16; s++) {
                const int k1 = t + T1 * s, lag = N2 * k1 + k2, at = 2 * pad16(k1);
                const float2 m2 = p2::fma(X[s], X[s], p2::mul(Y[s], Y[s]));
                const bool in = lag >= a.ws && lag < a.we;
                const bool ca = in && m2.x > a.t2, cb = in && live_b && m2.y > a.t2;
                if (!(ca || cb)) continue;
                const int bin = bin_of(lag - a.ws, bs, inv_bs);
                unsigned long long *key = keys + (g.kmod ? k1 * g.kmod + (bin & (g.kmod - 1)) : bin);
                if (ca) {
                  park[at] = make_float2(X[s].x, Y[s].x);
                  atomicMax(key, ((unsigned long long)(__float_as_uint(m2.x) & ~31u) << 32) | (unsigned)~lag);
                }
                if (cb) {
                  park[at + 1] = make_float2(X[s].y, Y[s].y);
                  atomicMax(key + nk, ((unsigned long long)(__float_as_uint(m2.y) & ~31u) << 32) | (unsigned)~lag);
                }
              }
            }
            __syncthreads();
            for (int b = tid; b < 2 * nk; b += 256) {
              const unsigned long long kk = keys[b];
              if (kk == 0ull) continue;
              keys[b] = 0ull;
              const int sel = b >= nk;
              const int lag = (int)(~(unsigned)kk), gw = (lag & (N2 - 1)) - k2base, k1w = lag / N2;
              const float2 v = reinterpret_cast<const float2 *>(buf + gw * ROW)[2 * pad16(k1w) + sel];
              rec_max(rec + sel * nb + bin_of(lag - a.ws, bs, inv_bs),
                      make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), (unsigned)kk, (unsigned)(kk >> 32)));
            }
            __syncthreads();          // the next unit's rows go where the values were parked
          }
        }
      }
    }
    __syncthreads();          // the ticket's writes are issued, its shared memory is free
    if (tid == 0) {
      if (tk.kind == L2_A) red_release32(a_done + slot);
      else {
        b_old = atom_add_acq_rel32(b_done + slot);
        b_item = tk.item;
      }
      next = atomicAdd(&g.ctl->ticket, 1ull);
    }
  }
  __syncthreads();
  if (tid == 0) {
    // low half: CTAs that left; high half: those that gave up
    const unsigned mine = gave_up ? 0x10001u : 1u;
    __threadfence();
    const unsigned sum = atomicAdd(&g.ctl->exits, mine) + mine;
    s_ok = (sum & 0xffffu) != gridDim.x ? 0 : (sum >> 16) ? 2 : 1;
  }
  __syncthreads();
  if (s_ok) {                 // every other CTA has left
    for (int i = tid; i < 3 * ring; i += 256) a_done[i] = 0u;
    if (s_ok == 2) {
      __threadfence();
      for (long long i = tid; i < (long long)ring * nb2; i += 256) g.rec[i] = make_uint4(0u, 0u, 0u, 0u);
      g.ctl->err = 0;
    }
    if (tid == 0) {
      g.ctl->ticket = 0ull;
      g.ctl->exits = 0u;
    }
  }
}

}  // namespace mfb
