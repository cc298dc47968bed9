// Radix-2/4/8/16 Stockham passes for two pairs per thread in packed FP32x2
// registers: X[i] = (re_A, re_B), Y[i] = (im_A, im_B) hold point i of pair A
// and of pair B, and every add, multiply or FMA is one FADD2 / FMUL2 / FFMA2.
// Operations, their order and their roundings are those of the one-pair
// passes (inverse_passes in flat_kernel.cuh), so both give the same bits.
#pragma once
#include "flat_kernel.cuh"

namespace mfb {

namespace p2 {

__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) {
  float2 r;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(*reinterpret_cast<unsigned long long *>(&r))
      : "l"(*reinterpret_cast<const unsigned long long *>(&a)),
        "l"(*reinterpret_cast<const unsigned long long *>(&b)));
  return r;
}
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }

// 2-point DFT on (X,Y)[O], (X,Y)[O + S].
template <int O, int S>
__device__ __forceinline__ void dft2(float2 *X, float2 *Y) {
  const float2 ax = X[O], ay = Y[O], bx = X[O + S], by = Y[O + S];
  X[O] = add(ax, bx);      Y[O] = add(ay, by);
  X[O + S] = sub(ax, bx);  Y[O + S] = sub(ay, by);
}

// 4-point inverse DFT on (X,Y)[O + S*q]; I2: input 2 is first multiplied by i.
// Scalar form: a = x0+x2, b = x0-x2, c = x1+x3, d = i(x1-x3); a+c, b+d, a-c, b-d.
template <int O, int S, bool I2 = false>
__device__ __forceinline__ void dft4(float2 *X, float2 *Y) {
  const float2 x0 = X[O], y0 = Y[O], x1 = X[O + S], y1 = Y[O + S];
  const float2 x3 = X[O + 3 * S], y3 = Y[O + 3 * S];
  float2 ax, ay, bx, by;
  if constexpr (I2) {   // x2 <- i * x2 = (-y2, x2)
    const float2 x2 = X[O + 2 * S], y2 = Y[O + 2 * S];
    ax = sub(x0, y2); ay = add(y0, x2);
    bx = add(x0, y2); by = sub(y0, x2);
  } else {
    const float2 x2 = X[O + 2 * S], y2 = Y[O + 2 * S];
    ax = add(x0, x2); ay = add(y0, y2);
    bx = sub(x0, x2); by = sub(y0, y2);
  }
  const float2 cx = add(x1, x3), cy = add(y1, y3);
  const float2 ex = sub(x1, x3), ey = sub(y1, y3);   // d = i*e = (-ey, ex)
  X[O] = add(ax, cx);          Y[O] = add(ay, cy);
  X[O + 2 * S] = sub(ax, cx);  Y[O + 2 * S] = sub(ay, cy);
  X[O + S] = sub(bx, ey);      Y[O + S] = add(by, ex);
  X[O + 3 * S] = add(bx, ey);  Y[O + 3 * S] = sub(by, ex);
}

// (X,Y)[i] *= exp(+2 pi i e / 16) for the exponents dft16 uses (e != 4).
template <int E>
__device__ __forceinline__ void tw16(float2 *X, float2 *Y, int i) {
  constexpr int e = E & 15;
  const float2 x = X[i], y = Y[i];
  if constexpr (e == 2) {
    X[i] = mul(dup(kSqrtHalf), sub(x, y));
    Y[i] = mul(dup(kSqrtHalf), add(x, y));
  } else if constexpr (e == 6) {
    X[i] = mul(dup(-kSqrtHalf), add(x, y));
    Y[i] = mul(dup(kSqrtHalf), sub(x, y));
  } else {
    static_assert(e == 1 || e == 3 || e == 9, "odd exponents of dft16");
    constexpr float c = (e == 1) ? kCos1_16 : (e == 3) ? kSin1_16 : -kCos1_16;
    constexpr float s = (e == 1) ? kSin1_16 : (e == 3) ? kCos1_16 : -kSin1_16;
    // scalar: {fmaf(x, c, -y*s), fmaf(x, s, y*c)}
    X[i] = fma(x, dup(c), mul(y, dup(-s)));
    Y[i] = fma(x, dup(s), mul(y, dup(c)));
  }
}

// 8-point inverse DFT on (X,Y)[O + S*q], natural order (the scalar dft8).
template <int O, int S>
__device__ __forceinline__ void dft8(float2 *X, float2 *Y) {
  dft4<O, 2 * S>(X, Y);
  dft4<O + S, 2 * S>(X, Y);
  tw16<2>(X, Y, O + 3 * S);
  tw16<6>(X, Y, O + 7 * S);
  float2 ax[4], ay[4], bx[4], by[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    ax[i] = X[O + 2 * i * S]; ay[i] = Y[O + 2 * i * S];
    bx[i] = X[O + (2 * i + 1) * S]; by[i] = Y[O + (2 * i + 1) * S];
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if (i == 2) {          // b2 = i * b = (-by, bx)
      X[O + i * S] = sub(ax[i], by[i]);        Y[O + i * S] = add(ay[i], bx[i]);
      X[O + (i + 4) * S] = add(ax[i], by[i]);  Y[O + (i + 4) * S] = sub(ay[i], bx[i]);
    } else {
      X[O + i * S] = add(ax[i], bx[i]);        Y[O + i * S] = add(ay[i], by[i]);
      X[O + (i + 4) * S] = sub(ax[i], bx[i]);  Y[O + (i + 4) * S] = sub(ay[i], by[i]);
    }
  }
}

// 16-point inverse DFT of (X,Y)[0..15], natural order (the scalar dft16).
__device__ __forceinline__ void dft16(float2 *X, float2 *Y) {
  dft4<0, 4>(X, Y);
  dft4<1, 4>(X, Y);
  dft4<2, 4>(X, Y);
  dft4<3, 4>(X, Y);
  tw16<1>(X, Y, 5);  tw16<2>(X, Y, 9);  tw16<3>(X, Y, 13);
  tw16<2>(X, Y, 6);                     tw16<6>(X, Y, 14);
  tw16<3>(X, Y, 7);  tw16<6>(X, Y, 11); tw16<9>(X, Y, 15);
  dft4<0, 1>(X, Y);
  dft4<4, 1>(X, Y);
  dft4<8, 1, true>(X, Y);    // slot 10 carries the twiddle i
  dft4<12, 1>(X, Y);
  float2 t;
#define P2_SWAP(a, b) t = X[a]; X[a] = X[b]; X[b] = t; t = Y[a]; Y[a] = Y[b]; Y[b] = t;
  P2_SWAP(1, 4) P2_SWAP(2, 8) P2_SWAP(3, 12) P2_SWAP(6, 9) P2_SWAP(7, 13) P2_SWAP(11, 14)
#undef P2_SWAP
}

// (X, Y) *= w for a twiddle w = (wr, wi) shared by both lanes, given as the
// record (wr, wr, wi, wi); scalar cmul: {fmaf(x, wr, -y*wi), fmaf(x, wi, y*wr)}.
__device__ __forceinline__ void twiddle(float2 &x, float2 &y, float4 w) {
  const float2 wr = make_float2(w.x, w.y), wi = make_float2(w.z, w.w);
  const float2 nx = fma(x, wr, mul(y, make_float2(-wi.x, -wi.y)));
  const float2 ny = fma(x, wi, mul(y, wr));
  x = nx;
  y = ny;
}

// Product of two twiddle records (both lanes carry the same value).
__device__ __forceinline__ float4 tw_mul(float4 a, float4 b) {
  float2 x = make_float2(a.x, a.y), y = make_float2(a.z, a.w);
  twiddle(x, y, b);
  return make_float4(x.x, x.y, y.x, y.y);
}

// Read-only 16-byte load kept inside the pair loop: the twiddle tables are
// loop-invariant, and hoisted into registers they would crowd out the
// transform's 64 values.
__device__ __forceinline__ float4 ldg4(const float4 *p) {
  float4 r;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
  return r;
}

// (X, Y)[q] *= w^q, q = 1..15, for one pass: w^1, w^2, w^3, w^4, w^8, w^12
// come from the FP64-built table (entry q at tw[(q-1)*stride]), the other
// nine are one product of two of those (w^(4a+b) = w^(4a) w^b), a rounding
// error of about one float ulp beside the table's half ulp.
__device__ __forceinline__ void pass_twiddles(float2 *X, float2 *Y, const float4 *tw, int stride) {
  const float4 w1 = ldg4(tw), w2 = ldg4(tw + stride), w3 = ldg4(tw + 2 * stride);
  const float4 w4 = ldg4(tw + 3 * stride), w8 = ldg4(tw + 7 * stride);
  const float4 w12 = ldg4(tw + 11 * stride);
  twiddle(X[1], Y[1], w1);
  twiddle(X[2], Y[2], w2);
  twiddle(X[3], Y[3], w3);
  twiddle(X[4], Y[4], w4);
  twiddle(X[5], Y[5], tw_mul(w4, w1));
  twiddle(X[6], Y[6], tw_mul(w4, w2));
  twiddle(X[7], Y[7], tw_mul(w4, w3));
  twiddle(X[8], Y[8], w8);
  twiddle(X[9], Y[9], tw_mul(w8, w1));
  twiddle(X[10], Y[10], tw_mul(w8, w2));
  twiddle(X[11], Y[11], tw_mul(w8, w3));
  twiddle(X[12], Y[12], w12);
  twiddle(X[13], Y[13], tw_mul(w12, w1));
  twiddle(X[14], Y[14], tw_mul(w12, w2));
  twiddle(X[15], Y[15], tw_mul(w12, w3));
}

// Inverse FFT of the N values (X, Y)[s] = x[t + T*s] of both pairs held by the
// T = N/16 threads of a transform (the packed inverse_passes); on return
// (X, Y)[q] = X[t + T*q].  Point i of the exchange sits at buf[pos(i)], one
// float4 (re_A, re_B, im_A, im_B) each; `sync` separates the transform's
// stores from its loads.  FIRST: synchronise before the first store (buf may
// still be read by the caller on entry); LAST: synchronise after the last load
// (buf is free again on return).
template <int N, bool FIRST, bool LAST, class Pos, class Sync>
__device__ __forceinline__ void passes(float2 *X, float2 *Y, float4 *buf, const float4 *twid, int t,
                                       Pos pos, Sync sync) {
  using Geo = FlatGeo<N>;
  constexpr int T = Geo::T, R0 = Geo::R0, PASSES = Geo::PASSES, B0 = 16 / R0;
  if constexpr (R0 == 16) dft16(X, Y);
  else if constexpr (R0 == 8) { dft8<0, 2>(X, Y); dft8<1, 2>(X, Y); }
  else if constexpr (R0 == 4) { dft4<0, 4>(X, Y); dft4<1, 4>(X, Y); dft4<2, 4>(X, Y); dft4<3, 4>(X, Y); }
  else {
    dft2<0, 8>(X, Y); dft2<1, 8>(X, Y); dft2<2, 8>(X, Y); dft2<3, 8>(X, Y);
    dft2<4, 8>(X, Y); dft2<5, 8>(X, Y); dft2<6, 8>(X, Y); dft2<7, 8>(X, Y);
  }
  if constexpr (FIRST) sync();
#pragma unroll
  for (int b = 0; b < B0; b++)
#pragma unroll
    for (int q = 0; q < R0; q++) {
      const int v = b + B0 * q;
      buf[pos((t + T * b) * R0 + q)] = make_float4(X[v].x, X[v].y, Y[v].x, Y[v].y);
    }
  sync();
#pragma unroll
  for (int p = 1; p < PASSES; p++) {
    const int Ns = span_before<N>(p);
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const float4 r = buf[pos(t + T * q)];
      X[q] = make_float2(r.x, r.y);
      Y[q] = make_float2(r.z, r.w);
    }
    const int k = t & (Ns - 1);
    pass_twiddles(X, Y, twid + twiddle_offset<N>(p) + k, Ns);
    dft16(X, Y);
    if (LAST || p < PASSES - 1) sync();
    if (p < PASSES - 1) {
      const int base = (t / Ns) * Ns * 16 + k;
#pragma unroll
      for (int q = 0; q < 16; q++)
        buf[pos(base + q * Ns)] = make_float4(X[q].x, X[q].y, Y[q].x, Y[q].y);
      sync();
    }
  }
}

}  // namespace p2

}  // namespace mfb
