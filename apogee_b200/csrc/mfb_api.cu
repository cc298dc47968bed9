// C ABI of libmfb.so: plans, ingest, launches.  See include/mfb.h.
//
// Host-side structure mirrors the reference engine (src/matchfilt.c for the
// flat plan, src/hmf.c for the hierarchical plan) but every hot loop is a
// device kernel on the plan's stream; the host only validates arguments and
// enqueues.  Nothing here allocates on the run path: buffers are sized at
// creation or grown on first use of a larger shape.
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdarg>
#include <cstring>
#include <cmath>
#include <string>
#include <vector>
#include <mutex>
#include <map>
#include <algorithm>
#include <memory>
#include <climits>
#include <cstddef>
#include "../../include/mfb.h"
#include "flat_kernel.cuh"
#include "flatw_kernel.cuh"
#include "series_kernel.cuh"
#include "hier_kernels.cuh"
#include "band_kernels.cuh"
#include "large_kernel.cuh"
#include "cluster_kernel.cuh"
#include "packed_passes.cuh"
#include "large2_kernel.cuh"
#include "adjoint_kernel.cuh"
#include "adjoint_direct.cuh"
#include "batch_kernel.cuh"
#include "gate_kernels.cuh"

using namespace mfb;

// ---------------------------------------------------------------- errors
static thread_local std::string g_err;

static int fail(int code, const char *fmt, ...) __attribute__((format(printf, 2, 3)));
static int fail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}
#define CUDA_TRY(expr)                                                              \
  do {                                                                              \
    cudaError_t _e = (expr);                                                        \
    if (_e != cudaSuccess)                                                          \
      return fail(MFB_ERR_CUDA, "%s: %s (%s:%d)", #expr, cudaGetErrorString(_e),    \
                  __FILE__, __LINE__);                                              \
  } while (0)

extern "C" const char *mfb_last_error(void) { return g_err.c_str(); }

// ------------------------------------------------------- twiddle tables
// exp(+2*pi*i*m/M), from double-precision cos/sin of a first-quadrant angle
// and an exact quadrant rotation, so that multiples of pi/2 come out as exact
// 0 and +-1 and the two components of pi/4 are equal.
static float2 unit_root(long long m, long long M) {
  m %= M;
  if (m < 0) m += M;
  const long long q4 = (4 * m) / M;          // quadrant
  const long long r = 4 * m - q4 * M;        // remainder, angle = (pi/2) * r / M
  double c0, s0;
  if (2 * r <= M) {
    const double th = M_PI / 2 * (double)r / (double)M;
    c0 = std::cos(th); s0 = std::sin(th);
  } else {
    const double th = M_PI / 2 * (double)(M - r) / (double)M;
    c0 = std::sin(th); s0 = std::cos(th);
  }
  if (r == 0) { c0 = 1.0; s0 = 0.0; }
  double c, s;
  switch (q4) {
    case 0: c = c0; s = s0; break;
    case 1: c = -s0; s = c0; break;
    case 2: c = -c0; s = -s0; break;
    default: c = s0; s = -c0; break;
  }
  return make_float2((float)c, (float)s);
}

template <int N>
static std::vector<float2> build_twiddles() {
  std::vector<float2> tw(twiddle_count<N>() > 0 ? twiddle_count<N>() : 1);
  for (int p = 1; p < FlatGeo<N>::PASSES; p++) {
    const int Ns = span_before<N>(p);
    const int off = twiddle_offset<N>(p);
    for (int q = 1; q < 16; q++)
      for (int k = 0; k < Ns; k++)
        tw[off + (q - 1) * Ns + k] = unit_root((long long)q * k, 16LL * Ns);
  }
  return tw;
}

// Per-(device, n) constant state: twiddles and launch shapes.
struct NConst {
  float2 *twid = nullptr;
  int grid_peaks = 0, grid_gate = 0, grid_fwd = 0;
  int cta = 0, smem = 0, g = 0;
  int grid_rows = 0;
  int grid_few = 0;             // items up to which flat_kernel runs one CTA per SM fewer
  // n = 128 ... 1024: the tables as (wr, wr, wi, wi) records for two pairs per
  // thread (the transforms of large2_kernel.cuh)
  float4 *twid2 = nullptr;
  // n >= 512: flatw_kernel's tables, in its thread order, and its grid
  float2 *twidw = nullptr;
  int gridw = 0, gridw_gate = 0;
};
static std::mutex g_const_mu;
static std::map<std::pair<int, int>, NConst> g_const;

template <int N>
static int make_const(int device, NConst &c) {
  using Geo = FlatGeo<N>;
  auto tw = build_twiddles<N>();
  CUDA_TRY(cudaMalloc(&c.twid, tw.size() * sizeof(float2)));
  CUDA_TRY(cudaMemcpy(c.twid, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice));
  c.cta = Geo::CTA;
  c.smem = Geo::SMEM;
  c.g = Geo::G;
  CUDA_TRY(cudaFuncSetAttribute(flat_kernel<N, MODE_PEAKS>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::SMEM));
  if constexpr (N < 512)
    CUDA_TRY(cudaFuncSetAttribute(flat_kernel<N, MODE_GATE>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::SMEM));
  CUDA_TRY(cudaFuncSetAttribute(series_forward_kernel<N>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::SMEM));
  CUDA_TRY(cudaFuncSetAttribute(rows_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                Geo::SMEM));
  int sms = 0, b1 = 0, b2 = 0, b3 = 0, b4 = 0;
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, flat_kernel<N, MODE_PEAKS>,
                                                         Geo::CTA, Geo::SMEM));
  if constexpr (N < 512)
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, flat_kernel<N, MODE_GATE>,
                                                           Geo::CTA, Geo::SMEM));
  else
    b2 = 1;   // flatw_kernel has the gate
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b3, series_forward_kernel<N>,
                                                         Geo::CTA, Geo::SMEM));
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b4, rows_kernel<N>, Geo::CTA,
                                                         Geo::SMEM));
  if (b1 < 1 || b2 < 1 || b3 < 1 || b4 < 1)
    return fail(MFB_ERR_CUDA, "kernel for n=%d cannot be resident on this device", N);
  if constexpr (N >= 128 && N <= 1024) {
    std::vector<float4> tw2(tw.size());
    for (size_t i = 0; i < tw.size(); i++) tw2[i] = make_float4(tw[i].x, tw[i].x, tw[i].y, tw[i].y);
    CUDA_TRY(cudaMalloc(&c.twid2, tw2.size() * sizeof(float4)));
    CUDA_TRY(cudaMemcpy(c.twid2, tw2.data(), tw2.size() * sizeof(float4), cudaMemcpyHostToDevice));
  }
  if constexpr (N >= 512) {
    using W = FlatWGeo<N>;
    std::vector<float2> t(W::TW);
    for (int i = 0; i < 15 * W::R; i++) t[i] = tw[i];
    for (int q = 0; q < 15; q++) {
      if (W::PASSES == 4)
        for (int K0 = 0; K0 < W::R; K0++)
          for (int K1 = 0; K1 < 16; K1++)
            t[W::OFF2 + q * 16 * W::R + 16 * K0 + K1] = tw[twiddle_offset<N>(2) + q * 16 * W::R + K0 + W::R * K1];
      for (int i = 0; i < W::T; i++) {
        const int k = W::PASSES == 3 ? (i >> 4) + W::R * (i & 15)
                                     : (i >> 8) + W::R * (((i >> 4) & 15) + 16 * (i & 15));
        t[W::OFF3 + q * W::T + i] = tw[twiddle_offset<N>(W::PASSES - 1) + q * W::T + k];
      }
    }
    CUDA_TRY(cudaMalloc(&c.twidw, t.size() * sizeof(float2)));
    CUDA_TRY(cudaMemcpy(c.twidw, t.data(), t.size() * sizeof(float2), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaFuncSetAttribute(flatw_kernel<N, MODE_PEAKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, W::SMEM));
    CUDA_TRY(cudaFuncSetAttribute(flatw_kernel<N, MODE_GATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, W::SMEM));
    int b5 = 0, b6 = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b5, flatw_kernel<N, MODE_PEAKS>, W::CTA, W::SMEM));
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b6, flatw_kernel<N, MODE_GATE>, W::CTA, W::SMEM));
    if (b5 < 1 || b6 < 1) return fail(MFB_ERR_CUDA, "block-bins kernel for n=%d cannot be resident", N);
    c.gridw = b5 * sms;
    c.gridw_gate = b6 * sms;
  }
  if constexpr (Geo::MINB > 1) {
    CUDA_TRY(cudaFuncSetAttribute(flat_kernel<N, MODE_PEAKS, Geo::MINB - 1>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::SMEM));
    c.grid_few = (Geo::MINB - 1) * sms;
  }
  c.grid_rows = b4 * sms;
  c.grid_peaks = b1 * sms;
  c.grid_gate = b2 * sms;
  c.grid_fwd = b3 * sms;
  return MFB_OK;
}

static int get_const(int device, int n, NConst **out) {
  std::lock_guard<std::mutex> lk(g_const_mu);
  auto key = std::make_pair(device, n);
  auto it = g_const.find(key);
  if (it != g_const.end()) { *out = &it->second; return MFB_OK; }
  NConst c;
  int r;
  switch (n) {
    case 64: r = make_const<64>(device, c); break;
    case 128: r = make_const<128>(device, c); break;
    case 256: r = make_const<256>(device, c); break;
    case 512: r = make_const<512>(device, c); break;
    case 1024: r = make_const<1024>(device, c); break;
    case 2048: r = make_const<2048>(device, c); break;
    case 4096: r = make_const<4096>(device, c); break;
    case 8192: r = make_const<8192>(device, c); break;
    case 16384: r = make_const<16384>(device, c); break;
    default: return fail(MFB_ERR_UNSUPPORTED, "unsupported transform length n=%d", n);
  }
  if (r != MFB_OK) return r;
  *out = &(g_const[key] = c);
  return MFB_OK;
}

// flatw_kernel covers n >= 512 with window and bins in whole blocks of n/16 lags
// (dense or listed), and every gate pass at those lengths; it gives the same bits
// as flat_kernel / rows_kernel.
static bool flatw_applies(int n, const NConst &c, const FlatArgs &a) {
  const int block = n / 16;
  return c.twidw && a.ws % block == 0 && a.we % block == 0 && a.binsize % block == 0;
}

template <int MODE>
static cudaError_t launch_flatw(int n, const NConst &c, FlatArgs a, cudaStream_t s) {
  a.twid = c.twidw;
  const int grid = MODE == MODE_PEAKS ? c.gridw : c.gridw_gate;
  switch (n) {
#define MFB_CASE(NN) \
  case NN: flatw_kernel<NN, MODE><<<grid, FlatWGeo<NN>::CTA, FlatWGeo<NN>::SMEM, s>>>(a); break;
    MFB_CASE(512) MFB_CASE(1024) MFB_CASE(2048) MFB_CASE(4096) MFB_CASE(8192) MFB_CASE(16384)
#undef MFB_CASE
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int N>
static void launch_peaks_n(const NConst &c, const FlatArgs &a, cudaStream_t s) {
  using Geo = FlatGeo<N>;
  if constexpr (Geo::MINB > 1) {
    const long long items = ((long long)a.nd * a.nt + Geo::G - 1) / Geo::G;
    if (items <= c.grid_few) {
      flat_kernel<N, MODE_PEAKS, Geo::MINB - 1><<<(int)items, Geo::CTA, Geo::SMEM, s>>>(a);
      return;
    }
  }
  flat_kernel<N, MODE_PEAKS><<<c.grid_peaks, Geo::CTA, Geo::SMEM, s>>>(a);
}

static cudaError_t launch_peaks(int n, const NConst &c, const FlatArgs &a, cudaStream_t s) {
  switch (n) {
#define MFB_CASE(NN) case NN: launch_peaks_n<NN>(c, a, s); break;
    MFB_CASE(64) MFB_CASE(128) MFB_CASE(256) MFB_CASE(512) MFB_CASE(1024)
    MFB_CASE(2048) MFB_CASE(4096) MFB_CASE(8192) MFB_CASE(16384)
#undef MFB_CASE
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

static cudaError_t launch_gate(int n, const NConst &c, const FlatArgs &a, cudaStream_t s) {
  switch (n) {
#define MFB_CASE(NN) case NN: flat_kernel<NN, MODE_GATE><<<c.grid_gate, c.cta, c.smem, s>>>(a); break;
    MFB_CASE(64) MFB_CASE(128) MFB_CASE(256)
#undef MFB_CASE
    default: return launch_flatw<MODE_GATE>(n, c, a, s);
  }
  return cudaGetLastError();
}

static cudaError_t launch_rows(int n, const NConst &c, const FlatArgs &a, cudaStream_t s) {
  switch (n) {
#define MFB_CASE(NN) case NN: rows_kernel<NN><<<c.grid_rows, c.cta, c.smem, s>>>(a); break;
    MFB_CASE(64) MFB_CASE(128) MFB_CASE(256) MFB_CASE(512) MFB_CASE(1024)
    MFB_CASE(2048) MFB_CASE(4096) MFB_CASE(8192) MFB_CASE(16384)
#undef MFB_CASE
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

static cudaError_t launch_forward(int n, const NConst &c, const SeriesArgs &a, cudaStream_t s) {
  switch (n) {
#define MFB_CASE(NN) case NN: series_forward_kernel<NN><<<c.grid_fwd, c.cta, c.smem, s>>>(a); break;
    MFB_CASE(64) MFB_CASE(128) MFB_CASE(256) MFB_CASE(512) MFB_CASE(1024)
    MFB_CASE(2048) MFB_CASE(4096) MFB_CASE(8192) MFB_CASE(16384)
#undef MFB_CASE
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

extern "C" int mfb_supported(size_t n) {
  return n >= 64 && n <= (1u << 20) && (n & (n - 1)) == 0;
}

static bool is_large(size_t n) { return n > 16384; }

// ------------------------------------------------------------ large-n setup
// n = N1 * N2 with N2 = 2^ceil(log2(n)/2) (<= 1024, the pass-A CTA size; two
// pass-A CTAs per SM at N2 = 512).
struct ClusterCfg {
  int C = 0, clusters = 0, clusters_small = 0, smem = 0;   // small: at most LARGE_SMALL_BINS bins
};
struct LargeConst {
  int N1 = 0, N2 = 0, lo_bits = 0;
  float2 *tw_hi = nullptr, *tw_lo = nullptr;
  NConst *c1 = nullptr, *c2 = nullptr;
  int grid_a = 0, grid_b = 0, smem_a = 0, smem_b = 0, cta_a = 0, cta_b = 0;
  int grid_bs = 0, smem_bs = 0;   // pass B with at most LARGE_SMALL_BINS keys
  // n = 32768 / 65536: one thread-block cluster per pair (cluster_kernel);
  // cl[0]: 256-thread CTAs, cl[1]: 512-thread CTAs
  ClusterCfg cl[2];
  // large2_kernel: pass-A twiddle anchors, units per item of both kinds, and its grid
  float2 *anchors = nullptr;
  int units_a = 0, units_b = 0, grid2 = 0;
};
static std::map<std::pair<int, int>, LargeConst> g_large;

// large2_kernel at every supported split.
#define LARGE2_SPLITS(X) X(128, 256) X(256, 256) X(256, 512) X(512, 512) X(512, 1024) X(1024, 1024)

constexpr int large2_smem(int nkeys) { return LARGE2_BUF * 16 + 2 * nkeys * 8; }

template <int N1, int N2>
static int large2_attr(LargeConst &c, int sms) {
  CUDA_TRY(cudaFuncSetAttribute(large2_kernel<N1, N2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                large2_smem(LARGE_MAX_BINS)));
  int b = 0;
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, large2_kernel<N1, N2>, 256,
                                                         large2_smem(LARGE_MAX_BINS)));
  if (b < 1) return fail(MFB_ERR_CUDA, "large kernel (%d x %d) cannot be resident", N1, N2);
  c.units_a = N1 / large2_cols<N2>();
  c.units_b = N2 / (256 / (N1 / 16));
  c.grid2 = 2 * sms;      // two CTAs per SM (registers, and shared memory but for some runs of many bins)
  LargeArgs a;
  memset(&a, 0, sizeof a);
  a.n = N1 * N2;
  a.tw_hi = c.tw_hi; a.tw_lo = c.tw_lo; a.lo_bits = c.lo_bits;
  CUDA_TRY(cudaMalloc(&c.anchors, (size_t)c.units_a * 5 * 256 * sizeof(float2)));
  large2_anchors<N2><<<c.units_a, 256>>>(a, c.anchors);
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaDeviceSynchronize());
  return MFB_OK;
}

template <int N2>
static int large_a_attr(int *grid, int *smem, int *cta, int sms) {
  *smem = LARGE_COLS * col_buf<N2>() * 8;
  *cta = N2;
  CUDA_TRY(cudaFuncSetAttribute(large_pass_a<N2>, cudaFuncAttributeMaxDynamicSharedMemorySize, *smem));
  CUDA_TRY(cudaFuncSetAttribute(large_fwd_a<N2>, cudaFuncAttributeMaxDynamicSharedMemorySize, *smem));
  int b = 0;
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, large_pass_a<N2>, *cta, *smem));
  if (b < 1) return fail(MFB_ERR_CUDA, "large pass A (N2=%d) cannot be resident", N2);
  *grid = b * sms;
  return MFB_OK;
}
template <int N1>
static int large_b_attr(LargeConst &c, int sms) {
  const int rows = FlatGeo<N1>::G * FlatGeo<N1>::BUF * 8;
  c.smem_b = rows + LARGE_MAX_BINS * 8;
  c.smem_bs = rows + LARGE_SMALL_BINS * 8;
  c.cta_b = FlatGeo<N1>::CTA;
  CUDA_TRY(cudaFuncSetAttribute(large_pass_b<N1>, cudaFuncAttributeMaxDynamicSharedMemorySize, c.smem_b));
  CUDA_TRY(cudaFuncSetAttribute(large_fwd_b<N1>, cudaFuncAttributeMaxDynamicSharedMemorySize, c.smem_b));
  int b = 0, bs = 0;
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, large_pass_b<N1>, c.cta_b, c.smem_b));
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bs, large_pass_b<N1>, c.cta_b, c.smem_bs));
  if (b < 1 || bs < 1) return fail(MFB_ERR_CUDA, "large pass B (N1=%d) cannot be resident", N1);
  c.grid_b = b * sms;
  c.grid_bs = bs * sms;
  return MFB_OK;
}

template <int N1, int N2, int C>
static void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, int clusters,
                           int smem, cudaStream_t s) {
  cfg = cudaLaunchConfig_t{};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(C * clusters);
  cfg.blockDim = dim3(ClusterGeo<N1, N2, C>::TH);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}

// Cluster kernel set-up for one geometry: shared memory, the non-portable
// cluster size 16 where it is used, and how many clusters fit at once.
template <int N1, int N2, int C>
static int cluster_attr(ClusterCfg &k) {
  using Geo = ClusterGeo<N1, N2, C>;
  k.smem = Geo::SMEM_FIXED + LARGE_MAX_BINS * 8;
  CUDA_TRY(cudaFuncSetAttribute(cluster_kernel<N1, N2, C>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
  if (C > 8)
    CUDA_TRY(cudaFuncSetAttribute(cluster_kernel<N1, N2, C>,
                                  cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  cluster_config<N1, N2, C>(cfg, at, 64, k.smem, nullptr);
  int n = 0, ns = 0;
  CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, cluster_kernel<N1, N2, C>, &cfg));
  cluster_config<N1, N2, C>(cfg, at, 64, Geo::SMEM_FIXED + LARGE_SMALL_BINS * 8, nullptr);
  CUDA_TRY(cudaOccupancyMaxActiveClusters(&ns, cluster_kernel<N1, N2, C>, &cfg));
  if (n < 1 || ns < 1) return fail(MFB_ERR_CUDA, "no cluster of %d CTAs fits for n=%d", C, N1 * N2);
  k.C = C;
  k.clusters = n;
  k.clusters_small = ns;
  return MFB_OK;
}

template <int N1, int N2, int C>
static cudaError_t launch_cluster_t(const LargeArgs &a, int clusters, int smem, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  cluster_config<N1, N2, C>(cfg, at, clusters, smem, s);
  return cudaLaunchKernelEx(&cfg, cluster_kernel<N1, N2, C>, a);
}

// One launch for every pair of the block or the list (no scratch, no host
// decision).  dense_pairs bounds the cluster count when the pairs are known.
static cudaError_t launch_cluster(const LargeConst &c, int mode, const LargeArgs &a,
                                  long long dense_pairs, cudaStream_t s) {
  const ClusterCfg &k = c.cl[mode - 1];
  const bool few = a.nb <= LARGE_SMALL_BINS;
  long long m = few ? k.clusters_small : k.clusters;
  if (dense_pairs > 0) m = std::min(m, dense_pairs);
  const int smem = k.smem - (LARGE_MAX_BINS - (few ? LARGE_SMALL_BINS : a.nb)) * 8;
  if (c.N1 == 128)
    return mode == 1 ? launch_cluster_t<128, 256, 8>(a, (int)m, smem, s)
                     : launch_cluster_t<128, 256, 4>(a, (int)m, smem, s);
  return mode == 1 ? launch_cluster_t<256, 256, 16>(a, (int)m, smem, s)
                   : launch_cluster_t<256, 256, 8>(a, (int)m, smem, s);
}

static int get_large(int device, int n, LargeConst **out) {
  {
    std::lock_guard<std::mutex> lk(g_const_mu);
    auto it = g_large.find({device, n});
    if (it != g_large.end()) { *out = &it->second; return MFB_OK; }
  }
  int L = 0;
  while ((1 << L) < n) L++;
  LargeConst c;
  c.N2 = 1 << ((L + 1) / 2);
  c.N1 = n / c.N2;
  c.lo_bits = (L + 1) / 2;
  int r = get_const(device, c.N1, &c.c1);
  if (r == MFB_OK) r = get_const(device, c.N2, &c.c2);
  if (r) return r;
  std::vector<float2> hi((size_t)n >> c.lo_bits), lo((size_t)1 << c.lo_bits);
  for (size_t i = 0; i < hi.size(); i++) hi[i] = unit_root((long long)(i << c.lo_bits), n);
  for (size_t i = 0; i < lo.size(); i++) lo[i] = unit_root((long long)i, n);
  CUDA_TRY(cudaMalloc(&c.tw_hi, hi.size() * sizeof(float2)));
  CUDA_TRY(cudaMalloc(&c.tw_lo, lo.size() * sizeof(float2)));
  CUDA_TRY(cudaMemcpy(c.tw_hi, hi.data(), hi.size() * sizeof(float2), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(c.tw_lo, lo.data(), lo.size() * sizeof(float2), cudaMemcpyHostToDevice));
  int sms = 0;
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  switch (c.N2) {
    case 256: r = large_a_attr<256>(&c.grid_a, &c.smem_a, &c.cta_a, sms); break;
    case 512: r = large_a_attr<512>(&c.grid_a, &c.smem_a, &c.cta_a, sms); break;
    case 1024: r = large_a_attr<1024>(&c.grid_a, &c.smem_a, &c.cta_a, sms); break;
    default: return fail(MFB_ERR_UNSUPPORTED, "no four-step split for n=%d", n);
  }
  if (r) return r;
  switch (c.N1) {
    case 128: r = large_b_attr<128>(c, sms); break;
    case 256: r = large_b_attr<256>(c, sms); break;
    case 512: r = large_b_attr<512>(c, sms); break;
    case 1024: r = large_b_attr<1024>(c, sms); break;
    default: return fail(MFB_ERR_UNSUPPORTED, "no four-step split for n=%d", n);
  }
  if (r) return r;
#define L2_CASE(A, B) if (c.N1 == A && c.N2 == B) r = large2_attr<A, B>(c, sms);
  LARGE2_SPLITS(L2_CASE)
#undef L2_CASE
  if (r) return r;
  if (n == 32768) {
    r = cluster_attr<128, 256, 8>(c.cl[0]);
    if (r == MFB_OK) r = cluster_attr<128, 256, 4>(c.cl[1]);
  } else if (n == 65536) {
    r = cluster_attr<256, 256, 16>(c.cl[0]);
    if (r == MFB_OK) r = cluster_attr<256, 256, 8>(c.cl[1]);
  }
  if (r) return r;
  std::lock_guard<std::mutex> lk(g_const_mu);
  *out = &(g_large[{device, n}] = c);
  return MFB_OK;
}

static cudaError_t launch_large(const LargeConst &c, const LargeArgs &a, cudaStream_t s) {
  switch (c.N2) {
    case 256: large_pass_a<256><<<c.grid_a, c.cta_a, c.smem_a, s>>>(a); break;
    case 512: large_pass_a<512><<<c.grid_a, c.cta_a, c.smem_a, s>>>(a); break;
    default: large_pass_a<1024><<<c.grid_a, c.cta_a, c.smem_a, s>>>(a); break;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const bool few = a.nb <= LARGE_SMALL_BINS;
  const int gb = few ? c.grid_bs : c.grid_b, sb = few ? c.smem_bs : c.smem_b;
  switch (c.N1) {
    case 128: large_pass_b<128><<<gb, c.cta_b, sb, s>>>(a); break;
    case 256: large_pass_b<256><<<gb, c.cta_b, sb, s>>>(a); break;
    case 512: large_pass_b<512><<<gb, c.cta_b, sb, s>>>(a); break;
    default: large_pass_b<1024><<<gb, c.cta_b, sb, s>>>(a); break;
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const long long outs = (long long)a.batch * a.nb;
  const int blocks = (int)std::min<long long>((outs + 255) / 256, 4096);
  large_finalize<<<blocks, 256, 0, s>>>(a);
  return cudaGetLastError();
}

static cudaError_t launch_large2(const LargeConst &c, const Large2Args &g, int grid, cudaStream_t s) {
  int smem = large2_smem(g.nkeys);
  // At N2 = 1024 a unit of kind A reads 32 bytes of every 128-byte line and finds the rest
  // in L1 later; two CTAs with this many keys would leave L1 20 KB (n = 2^20, 2 x 32 pairs,
  // 3000 bins: 831 us, one CTA per SM 624).
  if (c.N2 == 1024 && smem > 96 << 10) smem = std::max(smem, 116 << 10);
#define L2_CASE(A, B) if (c.N1 == A && c.N2 == B) large2_kernel<A, B><<<grid, 256, smem, s>>>(g);
  LARGE2_SPLITS(L2_CASE)
#undef L2_CASE
  return cudaGetLastError();
}

static cudaError_t launch_large_fwd(const LargeConst &c, const LargeArgs &a, const LargeFwd &f,
                                    cudaStream_t s) {
  switch (c.N2) {
    case 256: large_fwd_a<256><<<c.grid_a, c.cta_a, c.smem_a, s>>>(a, f); break;
    case 512: large_fwd_a<512><<<c.grid_a, c.cta_a, c.smem_a, s>>>(a, f); break;
    default: large_fwd_a<1024><<<c.grid_a, c.cta_a, c.smem_a, s>>>(a, f); break;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  switch (c.N1) {
    case 128: large_fwd_b<128><<<c.grid_bs, c.cta_b, c.smem_bs, s>>>(a, f); break;
    case 256: large_fwd_b<256><<<c.grid_bs, c.cta_b, c.smem_bs, s>>>(a, f); break;
    case 512: large_fwd_b<512><<<c.grid_bs, c.cta_b, c.smem_bs, s>>>(a, f); break;
    default: large_fwd_b<1024><<<c.grid_bs, c.cta_b, c.smem_bs, s>>>(a, f); break;
  }
  return cudaGetLastError();
}

extern "C" size_t mfb_nbins(size_t n, size_t binsize, size_t start, size_t end) {
  if (!binsize) return 0;
  if (end > n) end = n;
  if (start >= end) return 0;
  return (end - start + binsize - 1) / binsize;
}

// ---------------------------------------------------------------- flat plan
// large2_kernel's scratch, of one plan or shared (mfb_create_sharing): rows, and counters
// and candidate records.  The latter are zero between launches, whatever the plan
// and its layout of them, and are there twice: [0] for runs that follow one another and
// [1] for runs captured by a caller, whose order nobody here knows.
struct LargeScratch {
  int device;
  char *rows = nullptr, *state[2] = {nullptr, nullptr};   // one allocation, until state grows
  char *grown = nullptr;                                  // state's own, after that
  size_t rows_bytes = 0, state_bytes = 0;                 // state_bytes: each
  size_t refused = SIZE_MAX;                              // rows the device had no room for
  cudaEvent_t used = nullptr;         // after the last use outside a capture
  unsigned generation = 0;            // counts reallocations
  bool captured = false;              // a caller's graph may hold the present addresses
  std::vector<char *> kept;           // ... or these, outgrown since
  explicit LargeScratch(int dev) : device(dev) {}
  ~LargeScratch();
};

// Mapped host words for the error flags of large2_kernel launches, a page at a
// time and given back with the scratch that held them: page-locking memory for
// every plan would cost it about a millisecond.
static std::mutex g_err_mu;
static std::vector<int *> g_err_words;
static cudaError_t take_err_word(int **out) {
  std::lock_guard<std::mutex> lk(g_err_mu);
  if (g_err_words.empty()) {
    constexpr int WORDS = 1024;
    int *page = nullptr;
    cudaError_t e = cudaHostAlloc(&page, WORDS * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) return e;
    for (int i = 0; i < WORDS; i++) g_err_words.push_back(page + i);
  }
  *out = g_err_words.back();
  g_err_words.pop_back();
  **out = 0;
  return cudaSuccess;
}
static void give_err_word(int *w) {
  if (!w) return;
  std::lock_guard<std::mutex> lk(g_err_mu);
  g_err_words.push_back(w);
}

struct mfb_plan {
  int device = 0;
  size_t n = 0;
  int nd = 0, nt = 0;
  float2 *data = nullptr;   // [nd][n]
  float2 *tmpl = nullptr;   // [nt][n]
  cudaStream_t stream = nullptr;
  NConst *c = nullptr;
  // run_series workspace: block starts and block spectra
  uint64_t *starts_dev = nullptr;
  int starts_cap = 0;
  float2 *sspec = nullptr;
  int sspec_rows = 0;
  // large-n state: constants and scratch (empty until the first run that uses it)
  LargeConst *lc = nullptr;
  std::shared_ptr<LargeScratch> ls;
  int packed = 1;           // use flatw_kernel where it applies (mfb_set_packed)
  int cluster = -1;         // mfb_set_cluster's choice; -1: cluster_mode's rule
  int hold = 0;             // mfb_test_wait_limit
  bool own_capture = false; // a capture whose graph this library launches
  int *err = nullptr;       // mapped host word (g_err_words), set by a run that gave up
};

struct DeviceGuard {
  int prev = -1, dev_;
  explicit DeviceGuard(int dev) : dev_(dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() { if (prev >= 0 && prev != dev_) cudaSetDevice(prev); }
};

LargeScratch::~LargeScratch() {
  DeviceGuard dg(device);
  cudaFree(rows);
  cudaFree(grown);
  for (char *k : kept) cudaFree(k);
  if (used) cudaEventDestroy(used);
}

static int large_scratch(mfb_plan *p, long long pairs, size_t nb);
extern "C" int mfb_destroy(mfb_plan *p);
constexpr long long CLUSTER_PAIRS = 64;   // see cluster_mode
constexpr size_t EAGER_BINS = 512;        // 2 x 6.7 MB of records

// scratch: the large-n scratch to use, or nullptr for the plan's own; eager: allocate
// what a run without an allocation needs.
static int create_plan(mfb_plan **out, size_t n, int ndata, int ntmpl, int device,
                       const std::shared_ptr<LargeScratch> &scratch, bool eager) {
  if (!out) return fail(MFB_ERR_ARG, "null output handle");
  *out = nullptr;
  if (ndata < 1 || ntmpl < 1) return fail(MFB_ERR_ARG, "ndata and ntemplates must be >= 1");
  if (!mfb_supported(n))
    return fail(MFB_ERR_UNSUPPORTED,
                "unsupported matched-filter shape n=%zu ndata=%d ntemplates=%d", n, ndata, ntmpl);
  int ndev = 0;
  CUDA_TRY(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev) return fail(MFB_ERR_ARG, "no CUDA device %d", device);
  DeviceGuard dg(device);
  mfb_plan *p = new mfb_plan;
  p->device = device;
  p->n = n;
  p->nd = ndata;
  p->nt = ntmpl;
  int r = is_large(n) ? get_large(device, (int)n, &p->lc) : get_const(device, (int)n, &p->c);
  if (r != MFB_OK) { delete p; return r; }
  cudaError_t e1 = cudaMalloc(&p->data, (size_t)ndata * n * sizeof(float2));
  cudaError_t e2 = e1 == cudaSuccess ? cudaMalloc(&p->tmpl, (size_t)ntmpl * n * sizeof(float2)) : e1;
  if (e2 != cudaSuccess) {
    cudaFree(p->data);
    delete p;
    return fail(MFB_ERR_CUDA, "device allocation of %zu bytes failed: %s",
                ((size_t)ndata + ntmpl) * n * sizeof(float2), cudaGetErrorString(e2));
  }
  // Unset rows are zero spectra, not garbage.
  cudaMemset(p->data, 0, (size_t)ndata * n * sizeof(float2));
  cudaMemset(p->tmpl, 0, (size_t)ntmpl * n * sizeof(float2));
  CUDA_TRY(cudaDeviceSynchronize());
  if (is_large(n)) p->ls = scratch ? scratch : std::make_shared<LargeScratch>(device);
  if (eager && n == 32768 && (long long)ndata * ntmpl > CLUSTER_PAIRS) {
    // runs at this length do not allocate, up to EAGER_BINS bins (smaller blocks, lists and
    // captured runs take the cluster kernel, which has no scratch)
    r = large_scratch(p, (long long)ndata * ntmpl, EAGER_BINS);
    if (r != MFB_OK) { mfb_destroy(p); return r; }
  }
  *out = p;
  return MFB_OK;
}

extern "C" int mfb_create(mfb_plan **out, size_t n, int ndata, int ntmpl, int device) {
  return create_plan(out, n, ndata, ntmpl, device, nullptr, true);
}
extern "C" int mfb_create_sharing(mfb_plan **out, size_t n, int ndata, int ntmpl, mfb_plan *owner) {
  if (!owner) return fail(MFB_ERR_ARG, "null plan");
  return create_plan(out, n, ndata, ntmpl, owner->device, owner->ls, true);
}

extern "C" int mfb_destroy(mfb_plan *p) {
  if (!p) return MFB_OK;
  DeviceGuard dg(p->device);
  if (p->stream) cudaStreamSynchronize(p->stream); else cudaDeviceSynchronize();
  cudaFree(p->data);
  cudaFree(p->tmpl);
  cudaFree(p->starts_dev);
  cudaFree(p->sspec);
  p->ls.reset();
  give_err_word(p->err);
  delete p;
  return MFB_OK;
}

extern "C" int mfb_set_stream(mfb_plan *p, void *stream) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  p->stream = (cudaStream_t)stream;
  return MFB_OK;
}

static int copy_rows(float2 *dst, size_t n, int rows, int r0, int count, const void *src,
                     cudaStream_t s, const char *what) {
  if (!src) return fail(MFB_ERR_ARG, "null %s spectrum", what);
  if (count < 1 || r0 < 0 || r0 > rows - count)
    return fail(MFB_ERR_INDEX, "%s rows [%d, %d) out of range [0, %d)", what, r0, r0 + count, rows);
  CUDA_TRY(cudaMemcpyAsync(dst + (size_t)r0 * n, src, (size_t)count * n * sizeof(float2),
                           cudaMemcpyDefault, s));
  return MFB_OK;
}

extern "C" int mfb_set_data(mfb_plan *p, int d0, int count, const void *spec) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  DeviceGuard dg(p->device);
  return copy_rows(p->data, p->n, p->nd, d0, count, spec, p->stream, "data");
}

extern "C" int mfb_set_templates(mfb_plan *p, int t0, int count, const void *spec) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  DeviceGuard dg(p->device);
  return copy_rows(p->tmpl, p->n, p->nt, t0, count, spec, p->stream, "template");
}

// Validates a run's block, window and bins exactly as the reference binding
// does (python/matchedfilter/_core.c:29-43): returns nb or an error code.
static int check_run(const mfb_plan *p, int d0, int nd, int t0, int nt, size_t binsize,
                     size_t start, size_t end, size_t *nb) {
  if (d0 < 0 || nd < 1 || nd > p->nd || d0 > p->nd - nd || t0 < 0 || nt < 1 || nt > p->nt ||
      t0 > p->nt - nt || binsize < 1 || start >= p->n || end <= start)
    return fail(MFB_ERR_ARG, "invalid subrange, binsize or window");
  if (end > p->n) end = p->n;
  *nb = 1 + (end - start - 1) / binsize;
  return MFB_OK;
}

static FlatArgs base_args(const mfb_plan *p, int d0, int nd, int t0, int nt, size_t binsize,
                          float threshold, size_t start, size_t end, size_t nb) {
  FlatArgs a;
  memset(&a, 0, sizeof a);
  a.data = p->data;
  a.tmpl = p->tmpl;
  a.data_stride = (long long)p->n;
  a.tmpl_stride = (long long)p->n;
  a.twid = p->c ? p->c->twid : nullptr;
  a.d0 = d0; a.nd = nd; a.t0 = t0; a.nt = nt;
  if (end > p->n) end = p->n;
  a.ws = (int)start;
  a.we = (int)end;
  a.binsize = binsize > p->n ? (int)p->n : (int)binsize;   // one bin either way
  a.nb = (int)nb;
  a.t2 = threshold > 0.f ? threshold * threshold : 0.f;
  return a;
}

static bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return cs != cudaStreamCaptureStatusNone;
}
// Scratch of the large-n kernel, allocated on first use: a ring of item slots (two
// pairs each), two and a half times the kernel's delay between an item's two passes, or as
// many as the run has items if those are fewer (two at least), and records for the run's
// bins.  A run that needs more (run_series over many blocks, more bins) gets more; what it
// outgrows is freed, unless a caller's graph may hold it.  Under capture nothing is
// allocated: any ring of two slots or more will do.
static size_t large_ctl_bytes(int ring) {
  return (sizeof(Large2Ctl) + (size_t)ring * 3 * sizeof(unsigned) + 15) & ~(size_t)15;
}
static size_t large_state_bytes(int ring, size_t nb) {
  return large_ctl_bytes(ring) + (size_t)ring * 2 * nb * sizeof(uint4);
}
static int large_want(const mfb_plan *p, long long pairs) {
  const int per = (p->lc->units_a + p->lc->units_b) / LARGE2_GROUP;
  const long long most = large2_delay(p->lc->grid2, per) * 5 / 2;
  return (int)std::max<long long>(2, std::min((pairs + 1) / 2, most));
}
// Item slots of a run: what it wants, as far as the scratch has room.
static int large_ring(const mfb_plan *p, long long pairs, size_t nb) {
  const LargeScratch &s = *p->ls;
  int ring = (int)std::min<size_t>(large_want(p, pairs), s.rows_bytes / (p->n * sizeof(float4)));
  if (large_state_bytes(ring, nb) > s.state_bytes)
    ring = (int)((s.state_bytes - sizeof(Large2Ctl) - 16) / (3 * sizeof(unsigned) + 2 * nb * sizeof(uint4)));
  return ring;
}

// Whether a run of the plan gave up since the last look.
static int large_status(const mfb_plan *p) {
  if (!p->err || !*(volatile int *)p->err) return MFB_OK;
  *(volatile int *)p->err = 0;
  return fail(MFB_ERR_CUDA, "a run at n=%zu timed out on a dependency; its outputs are invalid", p->n);
}
// Keeps or frees an outgrown allocation.
static void large_drop(LargeScratch &s, char *block) {
  if (!block) return;
  if (s.captured) { s.kept.push_back(block); return; }
  cudaDeviceSynchronize();
  cudaFree(block);
}
static int large_scratch(mfb_plan *p, long long pairs, size_t nb) {
  if (int r = large_status(p)) return r;   // an earlier run gave up
  LargeScratch &s = *p->ls;
  const size_t slot = p->n * sizeof(float4);
  if (capturing(p->stream) && s.rows_bytes >= 2 * slot && s.state_bytes) return MFB_OK;
  const int ring = large_want(p, std::max(pairs, (long long)p->nd * p->nt));
  size_t rows = ring * slot;
  while (rows >= s.refused && rows > 2 * slot) rows = std::max(2 * slot, rows / 2);
  cudaError_t e = cudaSuccess;
  if (!s.used) e = cudaEventCreateWithFlags(&s.used, cudaEventDisableTiming);
  if (e == cudaSuccess && !p->err) e = take_err_word(&p->err);
  // records: as many as the bins ask for, two slots of LARGE_MAX_BINS at least
  const size_t state = std::max(std::max(large_state_bytes(ring, nb), large_state_bytes(2, LARGE_MAX_BINS)),
                                s.state_bytes);
  char *fresh = nullptr;
  if (e == cudaSuccess && s.rows_bytes < rows) {
    // one block for rows and state: an allocation costs a first run about 0.3 ms
    large_drop(s, s.rows);
    large_drop(s, s.grown);
    s.rows = s.grown = s.state[0] = s.state[1] = nullptr;
    s.rows_bytes = s.state_bytes = 0;
    s.captured = false;
    s.generation++;
    while ((e = cudaMalloc(&s.rows, rows + 2 * state)) == cudaErrorMemoryAllocation && rows > 2 * slot) {
      cudaGetLastError();             // a shorter ring is slower, no more
      s.refused = rows;
      rows = std::max(2 * slot, rows / 2);
    }
    if (e == cudaSuccess) {
      s.rows_bytes = rows;
      fresh = s.rows + rows;
    }
  } else if (e == cudaSuccess && s.state_bytes < state) {
    large_drop(s, s.grown);
    s.grown = s.state[0] = s.state[1] = nullptr;
    s.state_bytes = 0;
    s.generation++;
    e = cudaMalloc(&s.grown, 2 * state);
    fresh = s.grown;
  }
  if (e == cudaSuccess && fresh) {
    s.state[0] = fresh;
    s.state[1] = fresh + state;
    s.state_bytes = state;
    e = cudaMemset(fresh, 0, 2 * state);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();   // before any stream uses it
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(MFB_ERR_CUDA, "large-n scratch for n=%zu: %s", p->n, cudaGetErrorString(e));
  }
  return MFB_OK;
}
// Runs of one plan enqueued on different streams share its scratch: each waits
// for the one before.  A captured run is ordered by whoever launches its graph: by
// launch_hier_graph for the plan's own, else by the caller, who must not let it overlap
// another run of the plan.  If it does, both runs' outputs are wrong, but no later
// run's: a caller's captures have counters of their own, zeroed in front of each launch.
static cudaError_t scratch_begin(const mfb_plan *p) {
  return capturing(p->stream) ? cudaSuccess : cudaStreamWaitEvent(p->stream, p->ls->used, 0);
}
static cudaError_t scratch_end(const mfb_plan *p) {
  return capturing(p->stream) ? cudaSuccess : cudaEventRecord(p->ls->used, p->stream);
}
// Whether the plan's stream is being captured by a caller, whose graph then holds the
// scratch's addresses.
static bool note_capture(mfb_plan *p) {
  const bool foreign = capturing(p->stream) && !p->own_capture;
  if (foreign) p->ls->captured = true;
  return foreign;
}
// Series blocks that fit the scratch.
static int large_rows(const mfb_plan *p) { return (int)(p->ls->rows_bytes / (p->n * sizeof(float2))); }

constexpr int MANY_BINS = 1024;   // see short_run
// The cluster kernel's geometry for a run (1 or 2), or 0 for large2_kernel.  At
// n = 32768, unless mfb_set_cluster says otherwise, lists and dense runs of up to
// CLUSTER_PAIRS pairs take the cluster kernel (one cluster per pair has the
// shorter latency: 1 pair 16 against 19 us, 16 pairs 20 against 21, 51 listed rows
// of 4096 56 against 62), larger blocks large2_kernel (128 pairs 34 against
// 38 us, 1024 pairs 152 against 258).  `loose` bins (up to MANY_BINS of them, not shared by
// warps, at threshold 0) move the line to twice as many pairs: 96 pairs of 50 bins 38
// against 45 us in the launches per batch (short_run) and 50 in large2_kernel, 128 51
// against 51 and 57.  A captured run at that length keeps to the
// cluster kernel, which has no scratch: its graph may run beside other runs of the
// plan.
static int cluster_mode(const mfb_plan *p, bool listed, long long pairs, bool loose = false) {
  int mode = p->cluster;
  if (mode < 0)
    mode = p->n == 32768 && (listed || pairs <= (loose ? 2 : 1) * CLUSTER_PAIRS || capturing(p->stream)) ? 1 : 0;
  return mode > 0 && p->lc && p->lc->cl[mode - 1].C > 0 ? mode : 0;
}

// Short dense runs that take the launches per batch (pass A, pass B, finalize) instead of
// large2_kernel, whose ring neither fills nor overlaps the two passes on so few items:
// where bins are not whole multiples of N2 lags, either at threshold 0 (every lag a
// candidate) or with so many bins that writing them out counts; and a pair or two of the
// longest transform.  The limits, in lags of all pairs, are where the two meet.  B200, us here
// against large2_kernel, 1 x pairs: 50 ragged bins at threshold 0, n = 65536, 16 pairs 30 / 38,
// 128 92 / 98; n = 524288, 4 pairs 39 / 48; 4096 bins at threshold 0, n = 65536, 16 pairs 54 / 58, 32
// 81 / 63; above it, n = 65536, 8 pairs 22 / 35, 256 154 / 186, n = 131072, 256 323 / 275; n = 2^20, one
// pair 28 / 34.  Above a threshold with few bins large2_kernel wins from two pairs on
// (n = 65536, 16 pairs 24 / 19).
static bool short_run(const LargeArgs &a) {
  if (a.list) return false;
  if (a.n == 1 << 20 && a.total <= 2) return true;
  const long long points = a.total * a.n;
  if (a.seg > 0) return false;
  if (a.t2 > 0.f) return a.nb > MANY_BINS && points <= 1 << 24;
  return a.nb <= MANY_BINS ? points <= 1 << 23 : a.n <= 65536 && points <= 1 << 20;
}
// The launches per batch, in the scratch's rows, with the records of captured runs
// (zeroed here first).
static int run_batches(mfb_plan *p, LargeArgs a) {
  const LargeScratch &s = *p->ls;
  a.Y = reinterpret_cast<float2 *>(s.rows);
  a.rec = reinterpret_cast<uint4 *>(s.state[1]);
  note_capture(p);
  const int most = (int)std::min<size_t>(large_rows(p), s.state_bytes / ((size_t)a.nb * sizeof(uint4)));
  CUDA_TRY(scratch_begin(p));
  for (a.pair0 = 0; a.pair0 < a.total; a.pair0 += most) {
    a.batch = (int)std::min<long long>(most, a.total - a.pair0);
    CUDA_TRY(cudaMemsetAsync(a.rec, 0, (size_t)a.batch * a.nb * sizeof(uint4), p->stream));
    CUDA_TRY(launch_large(*p->lc, a, p->stream));
  }
  CUDA_TRY(scratch_end(p));
  return MFB_OK;
}

// list: listed rows; list_count: how many, on the device.  data: the rows to
// filter (default the plan's data rows).
static int run_large(mfb_plan *p, int d0, int nd, int t0, int nt, const int32_t *list,
                     const int32_t *list_count, size_t binsize, float threshold, size_t start,
                     size_t end, size_t nb, int64_t *idx, void *val, int32_t *counts, int rs,
                     const float2 *data = nullptr) {
  if (nb > (size_t)LARGE_MAX_BINS)
    return fail(MFB_ERR_UNSUPPORTED, "n=%zu supports at most %d bins per pair", p->n, LARGE_MAX_BINS);
  const LargeConst &c = *p->lc;
  const int bs = binsize > p->n ? (int)p->n : (int)binsize, seg = bin_lanes(bs, (int)start, c.N1, c.N2);
  const bool loose = seg == 0 && !(threshold > 0.f) && nb <= (size_t)MANY_BINS;
  const int cl = cluster_mode(p, list != nullptr, (long long)nd * nt, loose);
  if (!cl) {
    int sr = large_scratch(p, (long long)nd * nt, nb);
    if (sr) return sr;
  }
  if (end > p->n) end = p->n;
  LargeArgs a;
  memset(&a, 0, sizeof a);
  a.data = data ? data : p->data;
  a.tmpl = p->tmpl;
  a.n = (int)p->n; a.N1 = c.N1; a.N2 = c.N2;
  a.d0 = d0; a.nd = nd; a.t0 = t0; a.nt = nt;
  a.list = list;
  a.list_count = list ? list_count : nullptr;
  a.total = (long long)nd * nt;
  a.tw1 = c.c1->twid;
  a.tw2 = c.c2->twid;
  a.tw_hi = c.tw_hi;
  a.tw_lo = c.tw_lo;
  a.lo_bits = c.lo_bits;
  a.ws = (int)start; a.we = (int)end;
  a.binsize = bs;
  a.nb = (int)nb;
  a.seg = seg;
  a.t2 = threshold > 0.f ? threshold * threshold : 0.f;
  a.out_idx = (long long *)idx;
  a.out_val = (float2 *)val;
  a.rs = rs;
  a.out_cnt = counts;
  if (cl) {
    CUDA_TRY(launch_cluster(c, cl, a, list ? 0 : a.total, p->stream));
    return MFB_OK;
  }
  if (short_run(a)) return run_batches(p, a);
  Large2Args g;
  memset(&g, 0, sizeof g);
  g.a = a;
  g.tw1 = c.c1->twid2;
  g.tw2 = c.c2->twid2;
  g.anchors = c.anchors;
  g.Y = reinterpret_cast<float4 *>(p->ls->rows);
  const int foreign = note_capture(p);
  g.ring = large_ring(p, list ? LLONG_MAX - 1 : a.total, nb);
  g.ctl = reinterpret_cast<Large2Ctl *>(p->ls->state[foreign]);
  g.rec = reinterpret_cast<uint4 *>(p->ls->state[foreign] + large_ctl_bytes(g.ring));
  CUDA_TRY(cudaHostGetDevicePointer((void **)&g.err, p->err, 0));
  large2_keys(c.N1, 256 / (c.N1 / 16), a.binsize, a.ws, (int)nb, g.nkeys, g.kmod);
  g.spin = p->hold ? 1u << 14 : LARGE2_SPIN;
  g.hold = p->hold;
  const long long items = (a.total + 1) / 2;
  const int grid = (int)std::min<long long>(c.grid2, std::max<long long>(1, items * c.units_a));
  CUDA_TRY(scratch_begin(p));
  if (foreign) CUDA_TRY(cudaMemsetAsync(g.ctl, 0, large_state_bytes(g.ring, nb), p->stream));
  CUDA_TRY(launch_large2(c, g, grid, p->stream));
  CUDA_TRY(scratch_end(p));
  return MFB_OK;
}

// The dense block of `a` at n <= 16384.
static cudaError_t launch_dense(const mfb_plan *p, const FlatArgs &a) {
  if (p->packed && flatw_applies((int)p->n, *p->c, a))
    return launch_flatw<MODE_PEAKS>((int)p->n, *p->c, a, p->stream);
  return launch_peaks((int)p->n, *p->c, a, p->stream);
}

static int run_impl(mfb_plan *p, int d0, int nd, int t0, int nt, size_t binsize,
                    float threshold, size_t start, size_t end, int64_t *idx, void *val,
                    int32_t *counts, int rs) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  size_t nb;
  int r = check_run(p, d0, nd, t0, nt, binsize, start, end, &nb);
  if (r) return r;
  if (!idx || !val) return fail(MFB_ERR_ARG, "null output");
  if (std::isnan(threshold)) return fail(MFB_ERR_ARG, "threshold is NaN");
  DeviceGuard dg(p->device);
  FlatArgs a = base_args(p, d0, nd, t0, nt, binsize, threshold, start, end, nb);
  a.out_idx = (long long *)idx;
  a.out_val = (float2 *)val;
  a.rs = rs;
  a.out_cnt = counts;
  if (counts) CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)nd * nt * sizeof(int32_t), p->stream));
  if (is_large(p->n))
    return run_large(p, d0, nd, t0, nt, nullptr, nullptr, binsize, threshold, start, end, nb, idx, val,
                     counts, rs);
  CUDA_TRY(launch_dense(p, a));
  return MFB_OK;
}

extern "C" int mfb_status(mfb_plan *p) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  return large_status(p);
}
extern "C" int mfb_test_wait_limit(mfb_plan *p, int delta) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  if (!is_large(p->n)) return fail(MFB_ERR_STATE, "n=%zu has no pass to hold back", p->n);
  if (delta != 1 && delta != -1) return fail(MFB_ERR_ARG, "delta must be +1 or -1");
  p->hold += delta;
  return MFB_OK;
}
extern "C" int mfb_set_cluster(mfb_plan *p, int mode) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  if (mode < 0 || mode > 2) return fail(MFB_ERR_ARG, "cluster mode must be 0, 1 or 2");
  p->cluster = mode;
  return MFB_OK;
}

extern "C" int mfb_set_packed(mfb_plan *p, int on) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  p->packed = on ? 1 : 0;
  return MFB_OK;
}

extern "C" int mfb_run(mfb_plan *p, int d0, int nd, int t0, int nt, size_t binsize,
                       float threshold, size_t start, size_t end, int64_t *idx, void *val,
                       int32_t *counts) {
  return run_impl(p, d0, nd, t0, nt, binsize, threshold, start, end, idx, val, counts, 1);
}

extern "C" int mfb_run_records(mfb_plan *p, int d0, int nd, int t0, int nt, size_t binsize,
                               float threshold, size_t start, size_t end, void *records,
                               int32_t *counts) {
  if (!records) return fail(MFB_ERR_ARG, "null output");
  return run_impl(p, d0, nd, t0, nt, binsize, threshold, start, end, (int64_t *)records,
                  (char *)records + 8, counts, 2);
}

// trig_total: if set, the listed launch adds the row count to it on the
// device (the large-n path leaves it to the caller: returns 1 in *added = 0).
static int run_rows_impl(mfb_plan *p, int d0, int nd, int t0, int nt, const int32_t *rows,
                         const int32_t *nrows, int max_rows, size_t binsize, float threshold,
                         size_t start, size_t end, int64_t *idx, void *val, int32_t *counts,
                         int rs, unsigned long long *trig_total = nullptr, bool *added = nullptr,
                         int4 *host_rec = nullptr, bool *host_written = nullptr,
                         bool empty = false) {
  if (added) *added = false;
  if (host_written) *host_written = false;
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  size_t nb;
  int r = check_run(p, d0, nd, t0, nt, binsize, start, end, &nb);
  if (r) return r;
  if (!idx || !val || !rows || !nrows) return fail(MFB_ERR_ARG, "null pointer argument");
  if (max_rows < 0) return fail(MFB_ERR_ARG, "max_rows must be >= 0");
  DeviceGuard dg(p->device);
  FlatArgs a = base_args(p, d0, nd, t0, nt, binsize, threshold, start, end, nb);
  a.list = rows;
  a.list_count = nrows;
  a.out_idx = (long long *)idx;
  a.out_val = (float2 *)val;
  a.rs = rs;
  a.out_cnt = counts;   // rows not listed keep whatever the caller put there
  if (is_large(p->n) && empty && nb <= (size_t)LARGE_MAX_BINS) return large_status(p);
  if (is_large(p->n))
    return run_large(p, d0, nd, t0, nt, rows, nrows, binsize, threshold, start, end, nb, idx, val,
                     counts, rs);
  a.trig_total = trig_total;
  // more bins than key slots are stored lane by lane, too scattered for the host link
  // (n = 4096, 128 bins, 3277 rows: 436 us, hier_write_kernel after the refine 320)
  if (host_rec && rs == 2 && nb <= (size_t)KEYCAP) {
    a.host_rec = host_rec;
    if (host_written) *host_written = true;
  }
  if (p->packed && flatw_applies((int)p->n, *p->c, a)) {
    CUDA_TRY(launch_flatw<MODE_PEAKS>((int)p->n, *p->c, a, p->stream));
  } else {
    CUDA_TRY(launch_rows((int)p->n, *p->c, a, p->stream));
  }
  if (added) *added = trig_total != nullptr;
  return MFB_OK;
}

extern "C" int mfb_run_rows(mfb_plan *p, int d0, int nd, int t0, int nt, const int32_t *rows,
                            const int32_t *nrows, int max_rows, size_t binsize, float threshold,
                            size_t start, size_t end, int64_t *idx, void *val, int32_t *counts) {
  bool empty = false;
  if (p && is_large(p->n) && !cluster_mode(p, true, 0) && rows && nrows && max_rows >= 0) {
    // this length checks the list's length against max_rows: read it on the host
    DeviceGuard dg(p->device);
    int32_t cnt = 0;
    CUDA_TRY(cudaMemcpyAsync(&cnt, nrows, sizeof cnt, cudaMemcpyDeviceToHost, p->stream));
    CUDA_TRY(cudaStreamSynchronize(p->stream));
    if (cnt > max_rows) return fail(MFB_ERR_ARG, "row count %d exceeds max_rows %d", cnt, max_rows);
    empty = cnt == 0;
  }
  return run_rows_impl(p, d0, nd, t0, nt, rows, nrows, max_rows, binsize, threshold, start, end,
                       idx, val, counts, 1, nullptr, nullptr, nullptr, nullptr, empty);
}

extern "C" int mfb_forward(mfb_plan *p, const void *series, size_t nseries,
                           const uint64_t *starts_dev, int nblocks, void *spectra) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  if (!series || !starts_dev || !spectra || nblocks < 1)
    return fail(MFB_ERR_ARG, "invalid forward-transform arguments");
  DeviceGuard dg(p->device);
  if (is_large(p->n)) {
    int sr = large_scratch(p, nblocks, 1);
    if (sr) return sr;
    const LargeConst &c = *p->lc;
    LargeArgs a;
    memset(&a, 0, sizeof a);
    a.n = (int)p->n; a.N1 = c.N1; a.N2 = c.N2;
    a.total = nblocks;
    a.Y = reinterpret_cast<float2 *>(p->ls->rows);
    a.tw1 = c.c1->twid; a.tw2 = c.c2->twid;
    a.tw_hi = c.tw_hi; a.tw_lo = c.tw_lo; a.lo_bits = c.lo_bits;
    LargeFwd f;
    f.series = (const float2 *)series;
    f.nseries = (long long)nseries;
    f.starts = (const unsigned long long *)starts_dev;
    f.spectra = (float2 *)spectra;
    f.scale = 1.0f / (float)p->n;
    note_capture(p);
    CUDA_TRY(scratch_begin(p));
    for (long long p0 = 0; p0 < nblocks; p0 += large_rows(p)) {
      a.pair0 = p0;
      a.batch = (int)std::min<long long>(large_rows(p), nblocks - p0);
      CUDA_TRY(launch_large_fwd(c, a, f, p->stream));
    }
    CUDA_TRY(scratch_end(p));
    return MFB_OK;
  }
  SeriesArgs s;
  s.series = (const float2 *)series;
  s.nseries = (long long)nseries;
  s.starts = (const unsigned long long *)starts_dev;
  s.nblocks = nblocks;
  s.out = (float2 *)spectra;
  s.out_stride = (long long)p->n;
  s.twid = p->c->twid;
  s.scale = 1.0f / (float)p->n;
  CUDA_TRY(launch_forward((int)p->n, *p->c, s, p->stream));
  return MFB_OK;
}

// rs: stride of idx (int64) and val (complex64) between results, as FlatArgs has it.
static int run_series_impl(mfb_plan *p, const void *series, size_t nseries, const uint64_t *starts,
                           const uint64_t *win_start, const uint64_t *win_end, int nblocks, int t0,
                           int nt, size_t binsize, float threshold, int64_t *idx, void *val,
                           int32_t *counts, int rs) {
  if (!p) return fail(MFB_ERR_ARG, "null plan");
  if (!series || !starts || !win_start || !win_end || nblocks < 1 || !idx || !val)
    return fail(MFB_ERR_ARG, "invalid run_series arguments");
  if (t0 < 0 || nt < 1 || t0 > p->nt - nt || binsize < 1)
    return fail(MFB_ERR_ARG, "invalid template range or binsize");
  // Every window must give the same bin count (src/matchfilt.c:477-487).
  size_t nb0 = 0;
  for (int b = 0; b < nblocks; b++) {
    size_t lo = win_start[b], hi = win_end[b] > p->n ? p->n : win_end[b];
    if (lo >= hi || starts[b] > (uint64_t)INT64_MAX - p->n)
      return fail(MFB_ERR_ARG, "block %d has an empty window or an overflowing start", b);
    size_t nb = 1 + (hi - lo - 1) / binsize;
    if (b == 0) nb0 = nb;
    else if (nb != nb0) return fail(MFB_ERR_ARG, "block windows must have equal bin counts");
  }
  DeviceGuard dg(p->device);
  if (p->starts_cap < nblocks) {
    cudaFree(p->starts_dev);
    p->starts_dev = nullptr;
    p->starts_cap = 0;
    CUDA_TRY(cudaMalloc(&p->starts_dev, (size_t)nblocks * sizeof(uint64_t)));
    p->starts_cap = nblocks;
  }
  CUDA_TRY(cudaMemcpyAsync(p->starts_dev, starts, (size_t)nblocks * sizeof(uint64_t),
                           cudaMemcpyHostToDevice, p->stream));
  if (counts) CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)nblocks * nt * sizeof(int32_t), p->stream));
  // Block spectra go to a workspace of up to 64 MiB (at least one block),
  // grown on first use; the plan's data rows are left alone.
  const size_t row_bytes = p->n * sizeof(float2);
  int cap = (int)std::max<size_t>(1, ((size_t)64 << 20) / row_bytes);
  if (cap > nblocks) cap = nblocks;
  if (p->sspec_rows < cap) {
    cudaFree(p->sspec);
    p->sspec = nullptr;
    p->sspec_rows = 0;
    CUDA_TRY(cudaMalloc(&p->sspec, (size_t)cap * row_bytes));
    p->sspec_rows = cap;
  }
  if (is_large(p->n)) {   // the largest group's scratch at once
    int r = large_scratch(p, (long long)cap * nt, std::min<size_t>(nb0, LARGE_MAX_BINS));
    if (r) return r;
  }
  // Groups of consecutive equal windows, at most `cap` blocks each.
  for (int b0 = 0; b0 < nblocks;) {
    int g = 1;
    while (g < cap && b0 + g < nblocks && win_start[b0 + g] == win_start[b0] &&
           win_end[b0 + g] == win_end[b0])
      g++;
    int r = mfb_forward(p, series, nseries, p->starts_dev + b0, g, p->sspec);
    if (r) return r;
    size_t lo = win_start[b0], hi = win_end[b0];
    if (is_large(p->n)) {
      r = run_large(p, 0, g, t0, nt, nullptr, nullptr, binsize, threshold, lo, hi, nb0,
                    idx + (size_t)b0 * nt * nb0 * rs, (float2 *)val + (size_t)b0 * nt * nb0 * rs,
                    counts ? counts + (size_t)b0 * nt : nullptr, rs, p->sspec);
      if (r) return r;
      b0 += g;
      continue;
    }
    FlatArgs a = base_args(p, 0, g, t0, nt, binsize, threshold, lo, hi, nb0);
    a.data = p->sspec;
    a.out_idx = (long long *)idx + (size_t)b0 * nt * nb0 * rs;
    a.out_val = (float2 *)val + (size_t)b0 * nt * nb0 * rs;
    a.rs = rs;
    a.out_cnt = counts ? counts + (size_t)b0 * nt : nullptr;
    CUDA_TRY(launch_dense(p, a));
    b0 += g;
  }
  return MFB_OK;
}
extern "C" int mfb_run_series(mfb_plan *p, const void *series, size_t nseries,
                              const uint64_t *starts, const uint64_t *win_start,
                              const uint64_t *win_end, int nblocks, int t0, int nt,
                              size_t binsize, float threshold, int64_t *idx, void *val,
                              int32_t *counts) {
  return run_series_impl(p, series, nseries, starts, win_start, win_end, nblocks, t0, nt, binsize,
                         threshold, idx, val, counts, 1);
}
extern "C" int mfb_run_series_records(mfb_plan *p, const void *series, size_t nseries,
                                      const uint64_t *starts, const uint64_t *win_start,
                                      const uint64_t *win_end, int nblocks, int t0, int nt,
                                      size_t binsize, float threshold, void *records,
                                      int32_t *counts) {
  if (!records) return fail(MFB_ERR_ARG, "null pointer argument");
  return run_series_impl(p, series, nseries, starts, win_start, win_end, nblocks, t0, nt, binsize,
                         threshold, (int64_t *)records, (char *)records + 8, counts, 2);
}

// ---------------------------------------------------------- hierarchical plan
struct mfb_hplan {
  int device = 0;
  size_t n = 0, m = 0;
  int nd = 0, nt = 0;
  int kind = MFB_COARSE_FP32;
  mfb_plan *full = nullptr;     // full-length plan: data and templates at n
  float2 *ct = nullptr;         // coarse templates [nt][m] = H[:m] / sqrt(f)
  float *fpow = nullptr;        // per-template band fraction (float, as src/hmf.c:152)
  unsigned char *tready = nullptr;  // host flags: template row ingested
  NConst *cc = nullptr;         // constants at length m (FP32 coarse)
  int ref_on = 0;
  float ref_f = 0.f;
  float cal_thr = -1.f;
  int32_t *fire_list = nullptr; // [nd*nt]
  int32_t *fire_count = nullptr;// device counter
  unsigned long long *trig_total = nullptr;  // device: survivors summed over runs
  long long pairs = 0;
  TcCoarse *tc = nullptr;       // tensor-core coarse state
  // mfb_hier_run_host: which rows of the host table it last wrote hold refined
  // rows (marks, the last two lists, run parity; see hier_kernels.cuh)
  uint32_t *mark = nullptr;     // [nd*nt]
  int32_t *list_store = nullptr;// [2][nd*nt]
  int32_t *count_store = nullptr;
  unsigned *ctl = nullptr;
  const void *host_table = nullptr;
  long long host_rows = -1, host_nb = -1;
  // mfb_hier_run_host with host data: the bins above the band are copied on
  // a second stream while the coarse pass runs
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  // mfb_hier_run_host: the host-table bookkeeping runs on `side` beside the
  // refine, from ev_coarse (coarse pass done) to ev_table
  cudaEvent_t ev_coarse = nullptr, ev_table = nullptr;
  // mfb_hier_run_host repeated with identical arguments replays one CUDA
  // graph of the whole run (captured on `cap` at the second such call)
  struct RunKey {
    int d0, nd, t0, nt, same;
    uint32_t thr_bits, gate_bits;
    size_t binsize, start, end;
    const void *data, *records, *table, *info;
    unsigned scratch, pad;
  };
  RunKey last_key, graph_key;
  bool last_valid = false;
  cudaGraphExec_t graph = nullptr;
  cudaStream_t cap = nullptr;
  // band 16384 on the tensor cores (band_kernels.cuh): a batch of pairs'
  // 32 x 512 scratch, their row maxima, and the four-step's twiddles
  float2 *bY = nullptr;
  float *bM2 = nullptr;
  float2 *bw32 = nullptr, *bwm = nullptr;
  int bbatch = 0;
};

extern "C" int mfb_hier_create(mfb_hplan **out, size_t n, int ndata, int ntmpl, size_t band,
                               int coarse_kind, int device) {
  if (!out) return fail(MFB_ERR_ARG, "null output handle");
  *out = nullptr;
  if (!mfb_supported(n) || band < 64 || band >= n || (band & (band - 1)))
    return fail(MFB_ERR_UNSUPPORTED, "no hierarchical plan for n=%zu band=%zu", n, band);
  if (coarse_kind != MFB_COARSE_FP32 && coarse_kind != MFB_COARSE_BF16X3 &&
      coarse_kind != MFB_COARSE_FP16X3)
    return fail(MFB_ERR_ARG, "unknown coarse kind %d", coarse_kind);
  mfb_plan *full = nullptr;
  int r = create_plan(&full, n, ndata, ntmpl, device, nullptr, false);   // lists only
  if (r) return r;
  DeviceGuard dg(device);
  mfb_hplan *h = new mfb_hplan;
  h->device = device;
  h->n = n; h->m = band; h->nd = ndata; h->nt = ntmpl; h->kind = coarse_kind;
  h->full = full;
  h->tready = (unsigned char *)calloc((size_t)ntmpl, 1);
  r = get_const(device, (int)band, &h->cc);
  cudaError_t e = cudaSuccess;
  if (r == MFB_OK) {
    e = cudaMalloc(&h->ct, (size_t)ntmpl * band * sizeof(float2));
    if (e == cudaSuccess) e = cudaMalloc(&h->fpow, (size_t)ntmpl * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&h->fire_list, (size_t)ndata * ntmpl * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMalloc(&h->fire_count, sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMalloc(&h->trig_total, sizeof(unsigned long long));
    const size_t rows = (size_t)ndata * ntmpl;
    if (e == cudaSuccess) e = cudaMalloc(&h->mark, rows * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(h->mark, 0, rows * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&h->list_store, 2 * rows * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMalloc(&h->count_store, 2 * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMemset(h->count_store, 0, 2 * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMalloc(&h->ctl, 3 * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(h->ctl, 0, 3 * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_coarse, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_table, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->cap, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemset(h->trig_total, 0, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(h->ct, 0, (size_t)ntmpl * band * sizeof(float2));
    if (e == cudaSuccess) e = cudaMemset(h->fpow, 0, (size_t)ntmpl * sizeof(float));
  }
  if (r == MFB_OK && e == cudaSuccess && coarse_kind != MFB_COARSE_FP32) {
    if (band != (size_t)BAND_COLS && band != (size_t)BAND_BIG) {
      r = fail(MFB_ERR_UNSUPPORTED, "the tensor-core coarse pass covers band 512 and 16384, not %zu",
               band);
    } else {
      r = tc_coarse_create(&h->tc, BAND_COLS, ntmpl, ndata, coarse_kind == MFB_COARSE_FP16X3);
      if (r != 0) r = fail(MFB_ERR_CUDA, "tensor-core coarse setup failed: %s", tc_coarse_error());
    }
    if (r == MFB_OK && band == (size_t)BAND_BIG) {
      // 512 pairs per batch: a 64 MiB scratch that stays in L2 between the passes
      h->bbatch = (int)std::min<long long>(512, (long long)ndata * ntmpl);
      e = cudaMalloc(&h->bY, (size_t)h->bbatch * BAND_BIG * sizeof(float2));
      if (e == cudaSuccess) e = cudaMalloc(&h->bM2, (size_t)h->bbatch * BAND_ROWS * sizeof(float));
      if (e == cudaSuccess) e = cudaMalloc(&h->bw32, 16 * sizeof(float2));
      if (e == cudaSuccess) e = cudaMalloc(&h->bwm, 256 * sizeof(float2));
      if (e == cudaSuccess) {
        // W_16384^m = W^(128 (m >> 7)) * W^(m & 127): low table, then high table
        std::vector<float2> w32(16), wm(256);
        for (int k = 0; k < 16; k++) w32[k] = unit_root(k, BAND_ROWS);
        for (int i = 0; i < 128; i++) {
          wm[i] = unit_root(i, BAND_BIG);
          wm[128 + i] = unit_root(128LL * i, BAND_BIG);
        }
        e = cudaMemcpy(h->bw32, w32.data(), 16 * sizeof(float2), cudaMemcpyHostToDevice);
        if (e == cudaSuccess)
          e = cudaMemcpy(h->bwm, wm.data(), 256 * sizeof(float2), cudaMemcpyHostToDevice);
      }
    }
  }
  if (r != MFB_OK || e != cudaSuccess) {
    if (r == MFB_OK) r = fail(MFB_ERR_CUDA, "hierarchical plan allocation failed: %s",
                              cudaGetErrorString(e));
    mfb_hier_destroy(h);
    return r;
  }
  *out = h;
  return MFB_OK;
}

extern "C" int mfb_hier_destroy(mfb_hplan *h) {
  if (!h) return MFB_OK;
  DeviceGuard dg(h->device);
  cudaDeviceSynchronize();
  mfb_destroy(h->full);
  cudaFree(h->ct);
  cudaFree(h->fpow);
  cudaFree(h->fire_list);
  cudaFree(h->fire_count);
  cudaFree(h->trig_total);
  cudaFree(h->mark);
  cudaFree(h->list_store);
  cudaFree(h->count_store);
  cudaFree(h->ctl);
  if (h->side) cudaStreamDestroy(h->side);
  if (h->ev_fork) cudaEventDestroy(h->ev_fork);
  if (h->ev_join) cudaEventDestroy(h->ev_join);
  if (h->ev_coarse) cudaEventDestroy(h->ev_coarse);
  if (h->ev_table) cudaEventDestroy(h->ev_table);
  if (h->graph) cudaGraphExecDestroy(h->graph);
  if (h->cap) cudaStreamDestroy(h->cap);
  free(h->tready);
  tc_coarse_destroy(h->tc);
  cudaFree(h->bY);
  cudaFree(h->bM2);
  cudaFree(h->bw32);
  cudaFree(h->bwm);
  delete h;
  return MFB_OK;
}

// Forget the captured run and the repeated-call record: the next
// mfb_hier_run_host runs directly and captures again at the call after.
// Every plan input goes through the setters below, so a replay never runs
// with state that was changed after its capture.  (A graph still in flight
// is released by CUDA when it completes.)
static void hier_drop_graph(mfb_hplan *h) {
  h->last_valid = false;
  if (h->graph) {
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
}

extern "C" int mfb_hier_set_packed(mfb_hplan *h, int on) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  hier_drop_graph(h);
  return mfb_set_packed(h->full, on);
}

extern "C" int mfb_hier_set_cluster(mfb_hplan *h, int mode) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  hier_drop_graph(h);
  return mfb_set_cluster(h->full, mode);
}

extern "C" int mfb_hier_set_stream(mfb_hplan *h, void *stream) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  return mfb_set_stream(h->full, stream);
}

extern "C" int mfb_hier_set_data(mfb_hplan *h, int d0, int count, const void *spec) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  hier_drop_graph(h);
  return mfb_set_data(h->full, d0, count, spec);
}

// Rescale coarse templates for rows [t0, t0+count) from the plan's template
// bank: ct = H[:m] * (1/sqrt(f)) with f the reference fraction or each row's
// own band fraction (src/hmf.c:118-124,144-156).
static int refresh_coarse(mfb_hplan *h, int t0, int count) {
  HierScaleArgs s;
  s.tmpl = h->full->tmpl;
  s.n = (int)h->n;
  s.m = (int)h->m;
  s.t0 = t0;
  s.count = count;
  s.ref_on = h->ref_on;
  s.ref_f = h->ref_f;
  s.fpow = h->fpow;
  s.ct = h->ct;
  CUDA_TRY(launch_hier_scale(s, h->full->stream));
  if (h->tc) {
    int r = tc_coarse_pack_templates(h->tc, h->ct, t0, count, h->full->stream);
    if (r) return fail(MFB_ERR_CUDA, "tensor-core template pack failed: %s", tc_coarse_error());
  }
  return MFB_OK;
}

extern "C" int mfb_hier_set_templates(mfb_hplan *h, int t0, int count, const void *spec) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  int r = mfb_set_templates(h->full, t0, count, spec);
  if (r) return r;
  DeviceGuard dg(h->device);
  hier_drop_graph(h);
  HierFpowArgs f;
  f.tmpl = h->full->tmpl;
  f.n = (int)h->n;
  f.m = (int)h->m;
  f.t0 = t0;
  f.count = count;
  f.fpow = h->fpow;
  CUDA_TRY(launch_hier_fpow(f, h->full->stream));
  for (int t = t0; t < t0 + count; t++) h->tready[t] = 1;
  return refresh_coarse(h, t0, count);
}

extern "C" int mfb_hier_set_reference(mfb_hplan *h, const float *power) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  DeviceGuard dg(h->device);
  hier_drop_graph(h);
  if (power) {
    for (size_t k = 0; k < h->n; k++)
      if (!std::isfinite(power[k]) || power[k] < 0)
        return fail(MFB_ERR_ARG, "reference must be finite and nonnegative");
    double low = 0, total = 0;
    int rr = reference_fraction_fp64(power, h->n, h->m, &low, &total, h->full->stream);
    if (rr) return fail(MFB_ERR_CUDA, "reference sum failed: %s", cudaGetErrorString((cudaError_t)rr));
    if (!(total > 0)) return fail(MFB_ERR_ARG, "reference must have positive total power");
    h->ref_f = (float)(low / total);
    h->ref_on = 1;
  } else {
    h->ref_on = 0;
  }
  // Refresh every ingested template (contiguous runs of ready rows).
  for (int t = 0; t < h->nt;) {
    if (!h->tready[t]) { t++; continue; }
    int e = t;
    while (e < h->nt && h->tready[e]) e++;
    int r = refresh_coarse(h, t, e - t);
    if (r) return r;
    t = e;
  }
  return MFB_OK;
}

extern "C" int mfb_hier_set_threshold(mfb_hplan *h, float thr) {
  if (!h || !std::isfinite(thr)) return fail(MFB_ERR_ARG, "coarse threshold must be finite");
  if (thr != h->cal_thr) {
    DeviceGuard dg(h->device);
    hier_drop_graph(h);
  }
  h->cal_thr = thr;
  return MFB_OK;
}

// Coarse window on the lag grid R = n/m, widened by one coarse sample
// (src/hmf.c:233-239).
static void coarse_window(const mfb_hplan *h, size_t start, size_t end, int *cs, int *ce) {
  const size_t R = h->n / h->m;
  size_t cstart = start / R;
  size_t cend = (end + R - 1) / R;
  if (cend > h->m) cend = h->m;
  if (cstart > 0) cstart--;
  *cs = (int)cstart;
  *ce = (int)cend;
}

__global__ void accumulate_triggers(const int32_t *count, unsigned long long *total) {
  *total += (unsigned long long)*count;
}

// The band-16384 tensor-core coarse pass over the block (band_kernels.cuh):
// per batch of pairs, the column pass, the 512-point tensor-core pass over the
// scratch rows, and the per-pair maximum with the gate (or, with coarse_out,
// the coarse values).
static int band_big_coarse(mfb_hplan *h, int d0, int nd, int t0, int nt, int cs, int ce,
                           int64_t *idx, void *val, int rs, size_t full_nb, float *coarse_out,
                           cudaStream_t s) {
  mfb_plan *p = h->full;
  const long long total = (long long)nd * nt;
  int sms = 0;
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
  for (long long p0 = 0; p0 < total; p0 += h->bbatch) {
    const int batch = (int)std::min<long long>(h->bbatch, total - p0);
    BandColArgs c;
    c.data = p->data;
    c.data_stride = (long long)h->n;
    c.ct = h->ct;
    c.d0 = d0; c.nd = nd; c.t0 = t0; c.nt = nt;
    c.pair0 = p0;
    c.batch = batch;
    c.w32 = h->bw32;
    c.wm = h->bwm;
    c.Y = h->bY;
    const int gc = (int)std::min<long long>(2LL * batch, 8LL * sms);
    band_col_kernel<<<gc, 256, 0, s>>>(c);
    CUDA_TRY(cudaGetLastError());
    if (tc_coarse_rows(h->tc, h->bY, (long long)batch * BAND_ROWS, BAND_ROWS, cs, ce, h->bM2, s))
      return fail(MFB_ERR_CUDA, "tensor-core coarse pass failed: %s", tc_coarse_error());
    BandGateArgs g;
    g.m2 = h->bM2;
    g.pair0 = p0;
    g.batch = batch;
    g.nt = nt;
    g.total = total;
    g.t2 = h->cal_thr > 0.f ? h->cal_thr * h->cal_thr : 0.f;
    g.gate = h->cal_thr;
    g.out_idx = (long long *)idx;
    g.out_val = (float2 *)val;
    g.rs = rs;
    g.full_nb = (int)full_nb;
    g.fire_list = h->fire_list;
    g.fire_count = h->fire_count;
    g.coarse_out = coarse_out;
    band_gate_kernel<<<(batch + 7) / 8, 256, 0, s>>>(g);
    CUDA_TRY(cudaGetLastError());
  }
  return MFB_OK;
}

static int hier_run_impl(mfb_hplan *h, int d0, int nd, int t0, int nt, size_t binsize,
                         float threshold, size_t start, size_t end, int64_t *idx, void *val,
                         int32_t *counts, int rs, int phase = 0, void *table = nullptr,
                         long long *info = nullptr, const void *data_host = nullptr) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  mfb_plan *p = h->full;
  size_t nb;
  int r = check_run(p, d0, nd, t0, nt, binsize, start, end, &nb);
  if (r) return r;
  if (!idx || !val) return fail(MFB_ERR_ARG, "null output");
  if (!std::isfinite(h->cal_thr) || h->cal_thr < 0)
    return fail(MFB_ERR_STATE, "coarse threshold not configured");
  DeviceGuard dg(h->device);
  if (end > h->n) end = h->n;
  int cs, ce;
  coarse_window(h, start, end, &cs, &ce);
  cudaStream_t s = p->stream;
  bool join = false;
  if (data_host && phase == 0) {
    // all data rows from host memory: the band the coarse pass reads first,
    // the rest on the side stream, joined before the refine.  From pinned
    // memory the device gathers the band itself (one short launch instead of
    // a copy of nd strided rows); pageable memory takes the copy.
    const size_t row = h->n * sizeof(float2), band = h->m * sizeof(float2);
    cudaPointerAttributes pa;
    const bool mapped = cudaPointerGetAttributes(&pa, data_host) == cudaSuccess &&
                        pa.type == cudaMemoryTypeHost && pa.devicePointer != nullptr;
    if (!mapped) cudaGetLastError();
    if (mapped) {
      const float2 *src = (const float2 *)pa.devicePointer;
      const int elems = h->nd * (int)h->m;
      if ((((uintptr_t)src) & 15) == 0) {
        const int grid = std::max(1, std::min(1024, elems / 2 / 256));
        band_gather_kernel<2><<<grid, 256, 0, s>>>(p->data, (long long)h->n, src, (long long)h->n,
                                                   (int)h->m, h->nd);
      } else {
        const int grid = std::max(1, std::min(1024, elems / 256));
        band_gather_kernel<1><<<grid, 256, 0, s>>>(p->data, (long long)h->n, src, (long long)h->n,
                                                   (int)h->m, h->nd);
      }
      CUDA_TRY(cudaGetLastError());
    } else {
      CUDA_TRY(cudaMemcpy2DAsync(p->data, row, data_host, row, band, (size_t)h->nd,
                                 cudaMemcpyDefault, s));
    }
    CUDA_TRY(cudaEventRecord(h->ev_fork, s));
    CUDA_TRY(cudaStreamWaitEvent(h->side, h->ev_fork, 0));
    CUDA_TRY(cudaMemcpy2DAsync((char *)p->data + band, row, (const char *)data_host + band, row,
                               row - band, (size_t)h->nd, cudaMemcpyDefault, h->side));
    CUDA_TRY(cudaEventRecord(h->ev_join, h->side));
    join = true;
  }
  if (phase != 2) {
  CUDA_TRY(cudaMemsetAsync(h->fire_count, 0, sizeof(int32_t), s));
  if (counts) CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)nd * nt * sizeof(int32_t), s));
  if (h->kind == MFB_COARSE_FP32) {
    FlatArgs a;
    memset(&a, 0, sizeof a);
    a.data = p->data;
    a.tmpl = h->ct;
    a.data_stride = (long long)h->n;   // the first m bins of each full spectrum
    a.tmpl_stride = (long long)h->m;
    a.twid = h->cc->twid;
    a.d0 = d0; a.nd = nd; a.t0 = t0; a.nt = nt;
    a.ws = cs; a.we = ce; a.binsize = ce - cs; a.nb = 1;
    a.t2 = h->cal_thr > 0.f ? h->cal_thr * h->cal_thr : 0.f;
    a.out_idx = (long long *)idx;
    a.out_val = (float2 *)val;
    a.rs = rs;
    a.gate = h->cal_thr;
    a.fire_list = h->fire_list;
    a.fire_count = h->fire_count;
    a.full_nb = (int)nb;
    CUDA_TRY(launch_gate((int)h->m, *h->cc, a, s));
  } else if (h->m == (size_t)BAND_BIG) {
    r = band_big_coarse(h, d0, nd, t0, nt, cs, ce, idx, val, rs, nb, nullptr, s);
    if (r) return r;
  } else {
    TcRunArgs a;
    memset(&a, 0, sizeof a);
    a.data = p->data;
    a.ct = h->ct;
    a.n = (int)h->n;
    a.d0 = d0; a.nd = nd; a.t0 = t0; a.nt = nt;
    a.ws = cs; a.we = ce;
    a.gate = h->cal_thr;
    a.out_idx = (long long *)idx;
    a.out_val = (float2 *)val;
    a.rs = rs;
    a.full_nb = (int)nb;
    a.fire_list = h->fire_list;
    a.fire_count = h->fire_count;
    a.coarse_out = nullptr;
    int rr = tc_coarse_run(h->tc, a, s);
    if (rr) return fail(MFB_ERR_CUDA, "tensor-core coarse pass failed: %s", tc_coarse_error());
  }
  }
  if (phase == 1) return MFB_OK;
  // Host table: its bookkeeping (marks of this run's rows, reset of the
  // previous run's rows that are not refined now, list store, parity) needs
  // only the survivor list, so it runs on the second stream beside the refine.
  HierHostArgs ha;
  bool same = false;
  int hgrid = 1;
  const long long hrows = (long long)nd * nt;
  if (table) {
    ha.records = (const int4 *)idx;
    ha.table = (int4 *)table;
    ha.nb = (long long)nb;
    ha.list = h->fire_list;
    ha.count = h->fire_count;
    ha.mark = h->mark;
    ha.list_store = h->list_store;
    ha.count_store = h->count_store;
    ha.ctl = h->ctl;
    ha.rows = (long long)h->nd * h->nt;
    ha.total = h->trig_total;
    ha.info = info;
    ha.full_bytes = hrows * (long long)nb * 16;
    same = table == h->host_table && hrows == h->host_rows && (long long)nb == h->host_nb;
    ha.write_rows = same ? 1 : 0;
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
    hgrid = hier_host_grid(hrows * (long long)nb, sms);
    CUDA_TRY(cudaEventRecord(h->ev_coarse, s));
    CUDA_TRY(cudaStreamWaitEvent(h->side, h->ev_coarse, 0));
    hier_mark_kernel<<<hgrid, 256, 0, h->side>>>(ha);
    CUDA_TRY(cudaGetLastError());
    hier_unwrite_kernel<<<hgrid, 256, 0, h->side>>>(ha);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaEventRecord(h->ev_table, h->side));
  }
  if (join) CUDA_TRY(cudaStreamWaitEvent(s, h->ev_join, 0));
  // Refine the survivors with the full filter; no host decision in between.
  // With the host table as it was left by this plan, the single-block kernels also
  // store the refined rows into it.
  bool counted = false, host_written = false;
  r = run_rows_impl(p, d0, nd, t0, nt, h->fire_list, h->fire_count, nd * nt, binsize, threshold,
                    start, end, idx, val, counts, rs, table ? nullptr : h->trig_total, &counted,
                    table && same ? (int4 *)table : nullptr, &host_written);
  if (r) return r;
  if (table) {
    if (!same) CUDA_TRY(cudaMemcpyAsync(table, idx, (size_t)ha.full_bytes, cudaMemcpyDefault, s));
    else if (!host_written) {
      hier_write_kernel<<<hgrid, 256, 0, s>>>(ha);
      CUDA_TRY(cudaGetLastError());
    }
    CUDA_TRY(cudaStreamWaitEvent(s, h->ev_table, 0));
    h->host_table = table;
    h->host_rows = hrows;
    h->host_nb = (long long)nb;
  } else if (!counted) {
    accumulate_triggers<<<1, 1, 0, s>>>(h->fire_count, h->trig_total);
    CUDA_TRY(cudaGetLastError());
  }
  h->pairs += (long long)nd * nt;
  return MFB_OK;
}

extern "C" int mfb_hier_run(mfb_hplan *h, int d0, int nd, int t0, int nt, size_t binsize,
                            float threshold, size_t start, size_t end, int64_t *idx, void *val,
                            int32_t *counts) {
  return hier_run_impl(h, d0, nd, t0, nt, binsize, threshold, start, end, idx, val, counts, 1);
}

extern "C" int mfb_hier_run_phase(mfb_hplan *h, int phase, int d0, int nd, int t0, int nt,
                                  size_t binsize, float threshold, size_t start, size_t end,
                                  int64_t *idx, void *val, int32_t *counts) {
  if (phase < 0 || phase > 2) return fail(MFB_ERR_ARG, "phase must be 0, 1 or 2");
  return hier_run_impl(h, d0, nd, t0, nt, binsize, threshold, start, end, idx, val, counts, 1,
                       phase);
}

extern "C" int mfb_hier_run_records(mfb_hplan *h, int d0, int nd, int t0, int nt, size_t binsize,
                                    float threshold, size_t start, size_t end, void *records,
                                    int32_t *counts) {
  if (!records) return fail(MFB_ERR_ARG, "null output");
  return hier_run_impl(h, d0, nd, t0, nt, binsize, threshold, start, end, (int64_t *)records,
                       (char *)records + 8, counts, 2);
}

static uint32_t float_bits(float x) {
  uint32_t u;
  memcpy(&u, &x, sizeof u);
  return u;
}

// Launches the captured run, ordered with the plan's other runs as a direct run is.
static cudaError_t launch_hier_graph(mfb_hplan *h, cudaGraphExec_t x) {
  const mfb_plan *p = h->full;
  const bool ordered = p->ls && p->ls->used;
  cudaError_t e = ordered ? scratch_begin(p) : cudaSuccess;
  if (e == cudaSuccess) e = cudaGraphLaunch(x, p->stream);
  return e == cudaSuccess && ordered ? scratch_end(p) : e;
}

extern "C" int mfb_hier_run_host(mfb_hplan *h, int d0, int nd, int t0, int nt, size_t binsize,
                                 float threshold, size_t start, size_t end, const void *data,
                                 void *records, void *table, int64_t *info) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  if (!records || !table) return fail(MFB_ERR_ARG, "null output");
  if (((uintptr_t)records | (uintptr_t)table) & 15)
    return fail(MFB_ERR_ARG, "records and table must be 16-byte aligned");
  size_t nb;
  int r = check_run(h->full, d0, nd, t0, nt, binsize, start, end, &nb);
  if (r) return r;
  DeviceGuard dg(h->device);
  void *dtab = nullptr, *dinfo = nullptr;
  if (cudaHostGetDevicePointer(&dtab, table, 0) != cudaSuccess) {
    cudaGetLastError();
    return fail(MFB_ERR_ARG, "table must be pinned (page-locked, mapped) host memory");
  }
  if (info && cudaHostGetDevicePointer(&dinfo, info, 0) != cudaSuccess) {
    cudaGetLastError();
    return fail(MFB_ERR_ARG, "info must be pinned (page-locked, mapped) host memory");
  }
  // A graph may hold copies from pinned host memory only (a pageable copy is
  // synchronous and cannot be captured).
  bool graphable = true;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->full->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    graphable = false;   // the caller is capturing: record the kernels into its graph
  }
  if (data) {
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, data) != cudaSuccess) {
      cudaGetLastError();
      graphable = false;
    } else if (pa.type != cudaMemoryTypeHost) {
      graphable = false;
    }
  }
  r = large_status(h->full);   // an earlier run gave up
  if (r) return r;
  mfb_hplan::RunKey key;
  memset(&key, 0, sizeof key);
  key.d0 = d0; key.nd = nd; key.t0 = t0; key.nt = nt;
  key.same = dtab == h->host_table && (long long)nd * nt == h->host_rows &&
             (long long)nb == h->host_nb;
  key.thr_bits = float_bits(threshold);
  key.gate_bits = float_bits(h->cal_thr);
  key.binsize = binsize; key.start = start; key.end = end;
  key.data = data; key.records = records; key.table = dtab; key.info = dinfo;
  if (h->full->ls) key.scratch = h->full->ls->generation;   // a graph goes with its scratch
  if (graphable && h->graph && memcmp(&key, &h->graph_key, sizeof key) == 0) {
    CUDA_TRY(launch_hier_graph(h, h->graph));
    h->pairs += (long long)nd * nt;
    return MFB_OK;
  }
  const bool repeat = h->last_valid && memcmp(&key, &h->last_key, sizeof key) == 0;
  h->last_key = key;
  h->last_valid = false;
  if (graphable && repeat) {
    // second call with these arguments: capture the run once, replay it after
    // (the arguments equal the previous call's, so the host table is the
    // one this plan wrote last: the captured run is the changed-rows one)
    cudaStream_t user = h->full->stream;
    const long long pairs0 = h->pairs;
    h->full->stream = h->cap;
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    int rc = MFB_OK;
    cudaError_t e = cudaStreamBeginCapture(h->cap, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      h->full->own_capture = true;
      rc = hier_run_impl(h, d0, nd, t0, nt, binsize, threshold, start, end, (int64_t *)records,
                         (char *)records + 8, nullptr, 2, 0, dtab, (long long *)dinfo, data);
      h->full->own_capture = false;
      e = cudaStreamEndCapture(h->cap, &g);
    }
    h->full->stream = user;
    if (rc == MFB_OK && e == cudaSuccess && g) e = cudaGraphInstantiate(&x, g, 0);
    if (g) cudaGraphDestroy(g);
    if (rc == MFB_OK && e == cudaSuccess && x) {
      if (h->graph) cudaGraphExecDestroy(h->graph);
      h->graph = x;
      h->graph_key = key;
      CUDA_TRY(launch_hier_graph(h, x));
      h->last_valid = true;
      return MFB_OK;   // the captured call already counted its pairs
    }
    // capture failed: nothing ran; run the call directly
    if (x) cudaGraphExecDestroy(x);
    cudaGetLastError();
    h->pairs = pairs0;
  }
  r = hier_run_impl(h, d0, nd, t0, nt, binsize, threshold, start, end, (int64_t *)records,
                    (char *)records + 8, nullptr, 2, 0, dtab, (long long *)dinfo, data);
  if (r) {
    h->host_table = nullptr;
    return r;
  }
  h->last_valid = true;
  return MFB_OK;
}

extern "C" int mfb_hier_coarse_values(mfb_hplan *h, int d0, int nd, int t0, int nt, size_t start,
                                      size_t end, float *out) {
  if (!h || !out) return fail(MFB_ERR_ARG, "null argument");
  size_t nb;
  int r = check_run(h->full, d0, nd, t0, nt, 1, start, end, &nb);
  if (r) return r;
  DeviceGuard dg(h->device);
  if (end > h->n) end = h->n;
  int cs, ce;
  coarse_window(h, start, end, &cs, &ce);
  cudaStream_t s = h->full->stream;
  if (h->kind == MFB_COARSE_FP32) {
    FlatArgs a;
    memset(&a, 0, sizeof a);
    a.data = h->full->data;
    a.tmpl = h->ct;
    a.data_stride = (long long)h->n;
    a.tmpl_stride = (long long)h->m;
    a.twid = h->cc->twid;
    a.d0 = d0; a.nd = nd; a.t0 = t0; a.nt = nt;
    a.ws = cs; a.we = ce; a.binsize = ce - cs; a.nb = 1;
    a.t2 = 0.f;
    a.coarse_out = out;
    CUDA_TRY(launch_gate((int)h->m, *h->cc, a, s));
    return MFB_OK;
  }
  if (h->m == (size_t)BAND_BIG)
    return band_big_coarse(h, d0, nd, t0, nt, cs, ce, nullptr, nullptr, 1, 0, out, s);
  TcRunArgs a;
  memset(&a, 0, sizeof a);
  a.data = h->full->data;
  a.ct = h->ct;
  a.n = (int)h->n;
  a.d0 = d0; a.nd = nd; a.t0 = t0; a.nt = nt;
  a.ws = cs; a.we = ce;
  a.coarse_out = out;
  int rr = tc_coarse_run(h->tc, a, s);
  if (rr) return fail(MFB_ERR_CUDA, "tensor-core coarse pass failed: %s", tc_coarse_error());
  return MFB_OK;
}

// After a synchronisation: whether a coarse pass or a refine gave up.
static int hier_status(mfb_hplan *h) {
  if (tc_coarse_check(h->tc)) return fail(MFB_ERR_CUDA, "%s", tc_coarse_error());
  return large_status(h->full);
}

extern "C" int mfb_hier_status(mfb_hplan *h) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  return large_status(h->full);
}
extern "C" int mfb_hier_test_wait_limit(mfb_hplan *h, int delta) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  hier_drop_graph(h);
  return mfb_test_wait_limit(h->full, delta);
}

extern "C" int mfb_hier_last_triggers(mfb_hplan *h, int64_t *triggers) {
  if (!h || !triggers) return fail(MFB_ERR_ARG, "null argument");
  DeviceGuard dg(h->device);
  int32_t c = 0;
  CUDA_TRY(cudaMemcpyAsync(&c, h->fire_count, sizeof c, cudaMemcpyDeviceToHost, h->full->stream));
  CUDA_TRY(cudaStreamSynchronize(h->full->stream));
  if (int r = hier_status(h)) return r;
  *triggers = c;
  return MFB_OK;
}

extern "C" int mfb_hier_stats(mfb_hplan *h, int64_t *pairs, int64_t *triggers) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  DeviceGuard dg(h->device);
  unsigned long long tot = 0;
  CUDA_TRY(cudaMemcpyAsync(&tot, h->trig_total, sizeof tot, cudaMemcpyDeviceToHost, h->full->stream));
  CUDA_TRY(cudaStreamSynchronize(h->full->stream));
  if (int r = hier_status(h)) return r;
  if (pairs) *pairs = h->pairs;
  if (triggers) *triggers = (int64_t)tot;
  return MFB_OK;
}

extern "C" int mfb_hier_config(mfb_hplan *h, size_t *band, int *kind) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  if (band) *band = h->m;
  if (kind) *kind = h->kind;
  return MFB_OK;
}

// ------------------------------------------------------------ measurement
__global__ void fp32_fma_probe(float *out, int iters) {
  float a0 = threadIdx.x * 1e-3f, a1 = a0 + 1.f, a2 = a0 + 2.f, a3 = a0 + 3.f;
  float a4 = a0 + 4.f, a5 = a0 + 5.f, a6 = a0 + 6.f, a7 = a0 + 7.f;
  const float b = 0.999999f, c = 1e-7f;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int u = 0; u < 16; u++) {
      a0 = fmaf(a0, b, c); a1 = fmaf(a1, b, c); a2 = fmaf(a2, b, c); a3 = fmaf(a3, b, c);
      a4 = fmaf(a4, b, c); a5 = fmaf(a5, b, c); a6 = fmaf(a6, b, c); a7 = fmaf(a7, b, c);
    }
  }
  const float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == 12345.f) out[threadIdx.x] = s;   // keeps the loop live
}

extern "C" int mfb_fp32_peak(int device, double *flops_per_s) {
  if (!flops_per_s) return fail(MFB_ERR_ARG, "null output");
  DeviceGuard dg(device);
  int sms = 0;
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  float *out = nullptr;
  CUDA_TRY(cudaMalloc(&out, 1024 * sizeof(float)));
  const int threads = 1024, blocks = sms * 2, iters = 4096;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  fp32_fma_probe<<<blocks, threads>>>(out, iters);   // warm-up
  cudaEventRecord(e0);
  fp32_fma_probe<<<blocks, threads>>>(out, iters);
  cudaEventRecord(e1);
  cudaError_t e = cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return fail(MFB_ERR_CUDA, "probe failed: %s", cudaGetErrorString(e));
  const double fmas = (double)blocks * threads * iters * 16.0 * 8.0;
  *flops_per_s = 2.0 * fmas / (ms * 1e-3);
  return MFB_OK;
}

// ------------------------------------------ large transforms without allocation
// Some callers cannot let a library allocate device memory: a serving process
// that hands all of HBM to its own pool or arena at start-up leaves nothing for
// cudaMalloc, and a pipeline on a latency budget cannot absorb the device-wide
// synchronisation that cudaMalloc and cudaFree imply while its other streams
// run.  mfb_run_large_static serves them with the two-pass filter for large n:
// no plan, device inputs and outputs from the caller, and its scratch (the
// pass-A rows and the per-bin records) in the file-scope array below, reserved
// with the module.  Its twiddles sit in a second file-scope table, uploaded
// once per device by the set-up of the first call on that device.
constexpr int STATIC_MIN_LOG = 15, STATIC_MAX_LOG = 19;   // n = 32768 ... 524288
constexpr int kStaticFft[4] = {128, 256, 512, 1024};      // N1 and N2 of those n

constexpr int static_fft_count(int N) {
  return N == 128 ? twiddle_count<128>()
       : N == 256 ? twiddle_count<256>()
       : N == 512 ? twiddle_count<512>()
                  : twiddle_count<1024>();
}
// Offset of the inter-pass table of the N-point FFT.
constexpr int static_fft_off(int N) {
  int o = 0;
  for (int i = 0; i < 4 && kStaticFft[i] < N; i++) o += static_fft_count(kStaticFft[i]);
  return o;
}
// Offset of the W_n hi table of n = 2^L (its lo table follows it).
constexpr int static_root_off(int L) {
  int o = static_fft_off(2048);
  for (int l = STATIC_MIN_LOG; l < L; l++) o += (1 << (l - (l + 1) / 2)) + (1 << ((l + 1) / 2));
  return o;
}
constexpr int STATIC_TW_COUNT = static_root_off(STATIC_MAX_LOG + 1);

static __device__ __align__(256) unsigned char g_static_scratch[MFB_STATIC_SCRATCH_BYTES];
static __device__ __align__(256) float2 g_static_twiddles[STATIC_TW_COUNT];

struct StaticDev {
  bool ready = false;
  unsigned char *scratch = nullptr;     // device address of g_static_scratch
  float2 *tw = nullptr;                 // device address of g_static_twiddles
  LargeConst shape[STATIC_MAX_LOG + 1]; // launch shapes per log2(n)
};
constexpr int STATIC_MAX_DEVICES = 64;
static std::mutex g_static_mu;
static StaticDev g_static[STATIC_MAX_DEVICES];

// Once per device, with that device current: the symbol addresses, the twiddle
// upload and the kernel attributes.  Synchronous, so it must not run inside a
// stream capture.
static int static_setup(int device, StaticDev **out) {
  std::lock_guard<std::mutex> lk(g_static_mu);
  StaticDev &s = g_static[device];
  if (!s.ready) {
    void *ptr = nullptr;
    CUDA_TRY(cudaGetSymbolAddress(&ptr, g_static_scratch));
    s.scratch = (unsigned char *)ptr;
    CUDA_TRY(cudaGetSymbolAddress(&ptr, g_static_twiddles));
    s.tw = (float2 *)ptr;
    std::vector<float2> tw(STATIC_TW_COUNT);
    auto put = [&](int N, const std::vector<float2> &t) {
      std::copy(t.begin(), t.begin() + static_fft_count(N), tw.begin() + static_fft_off(N));
    };
    put(128, build_twiddles<128>());
    put(256, build_twiddles<256>());
    put(512, build_twiddles<512>());
    put(1024, build_twiddles<1024>());
    for (int L = STATIC_MIN_LOG; L <= STATIC_MAX_LOG; L++) {
      const int lo_bits = (L + 1) / 2, n = 1 << L;
      float2 *hi = tw.data() + static_root_off(L), *lo = hi + (n >> lo_bits);
      for (int i = 0; i < (n >> lo_bits); i++) hi[i] = unit_root((long long)i << lo_bits, n);
      for (int i = 0; i < (1 << lo_bits); i++) lo[i] = unit_root(i, n);
    }
    CUDA_TRY(cudaMemcpy(s.tw, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice));
    int sms = 0, r = MFB_OK;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    for (int L = STATIC_MIN_LOG; L <= STATIC_MAX_LOG && r == MFB_OK; L++) {
      LargeConst &c = s.shape[L];
      c.lo_bits = (L + 1) / 2;
      c.N2 = 1 << c.lo_bits;
      c.N1 = 1 << (L - c.lo_bits);
      switch (c.N2) {
        case 256: r = large_a_attr<256>(&c.grid_a, &c.smem_a, &c.cta_a, sms); break;
        case 512: r = large_a_attr<512>(&c.grid_a, &c.smem_a, &c.cta_a, sms); break;
        default: r = large_a_attr<1024>(&c.grid_a, &c.smem_a, &c.cta_a, sms); break;
      }
      if (r) break;
      switch (c.N1) {
        case 128: r = large_b_attr<128>(c, sms); break;
        case 256: r = large_b_attr<256>(c, sms); break;
        default: r = large_b_attr<512>(c, sms); break;
      }
    }
    if (r) return r;
    s.ready = true;
  }
  *out = &s;
  return MFB_OK;
}

extern "C" int mfb_run_large_static(int device, size_t n, const void *data, int nd,
                                    const void *templates, int nt, size_t binsize,
                                    float threshold, size_t start, size_t end, int64_t *idx,
                                    void *val, int32_t *counts, void *stream) {
  if (!data || !templates || !idx || !val) return fail(MFB_ERR_ARG, "null pointer");
  if (nd < 1 || nt < 1) return fail(MFB_ERR_ARG, "ndata and ntemplates must be >= 1");
  if (std::isnan(threshold)) return fail(MFB_ERR_ARG, "threshold is NaN");
  int L = 0;
  while (L < 62 && ((size_t)1 << L) < n) L++;
  if (((size_t)1 << L) != n || L < STATIC_MIN_LOG)
    return fail(MFB_ERR_UNSUPPORTED,
                "mfb_run_large_static: n=%zu is not a power of two >= 32768 (mfb_run covers it)", n);
  const size_t nb = mfb_nbins(n, binsize, start, end);
  if (nb == 0) return fail(MFB_ERR_ARG, "zero binsize or empty window [%zu, %zu)", start, end);
  if (nb > (size_t)LARGE_MAX_BINS)
    return fail(MFB_ERR_UNSUPPORTED, "mfb_run_large_static: %zu bins per pair; at most %d",
                nb, LARGE_MAX_BINS);
  const size_t rec_one = (nb * sizeof(uint4) + 255) & ~(size_t)255;
  const size_t need = rec_one + n * sizeof(float2);
  if (need > (size_t)MFB_STATIC_SCRATCH_BYTES || L > STATIC_MAX_LOG)
    return fail(MFB_ERR_UNSUPPORTED,
                "mfb_run_large_static: n=%zu needs %zu bytes of scratch for one pair; the static "
                "scratch holds %zu (MFB_STATIC_SCRATCH_BYTES)",
                n, need, (size_t)MFB_STATIC_SCRATCH_BYTES);
  int ndev = 0;
  CUDA_TRY(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev || device >= STATIC_MAX_DEVICES)
    return fail(MFB_ERR_ARG, "no device %d", device);
  DeviceGuard dg(device);
  StaticDev *s = nullptr;
  int r = static_setup(device, &s);
  if (r) return r;
  // Pairs per batch: records [batch][nb] first, then rows [batch][n].
  long long batch = (long long)(MFB_STATIC_SCRATCH_BYTES / (nb * sizeof(uint4) + n * sizeof(float2)));
  auto bytes = [&](long long b) {
    return ((b * nb * sizeof(uint4) + 255) & ~(size_t)255) + b * n * sizeof(float2);
  };
  while (batch > 1 && bytes(batch) > (size_t)MFB_STATIC_SCRATCH_BYTES) batch--;
  const long long total = (long long)nd * nt;
  if (batch > total) batch = total;
  const LargeConst &c = s->shape[L];
  uint4 *rec = reinterpret_cast<uint4 *>(s->scratch);
  float2 *Y = reinterpret_cast<float2 *>(s->scratch + ((batch * nb * sizeof(uint4) + 255) & ~(size_t)255));
  cudaStream_t st = (cudaStream_t)stream;
  if (end > n) end = n;
  LargeArgs a;
  memset(&a, 0, sizeof a);
  a.data = (const float2 *)data;
  a.tmpl = (const float2 *)templates;
  a.n = (int)n; a.N1 = c.N1; a.N2 = c.N2;
  a.d0 = 0; a.nd = nd; a.t0 = 0; a.nt = nt;
  a.list = nullptr;
  a.total = total;
  a.Y = Y;
  a.rec = rec;
  a.tw1 = s->tw + static_fft_off(c.N1);
  a.tw2 = s->tw + static_fft_off(c.N2);
  a.tw_hi = s->tw + static_root_off(L);
  a.tw_lo = a.tw_hi + (n >> c.lo_bits);
  a.lo_bits = c.lo_bits;
  a.ws = (int)start; a.we = (int)end;
  a.binsize = binsize > n ? (int)n : (int)binsize;
  a.nb = (int)nb;
  a.t2 = threshold > 0.f ? threshold * threshold : 0.f;
  a.out_idx = (long long *)idx;
  a.out_val = (float2 *)val;
  a.rs = 1;
  a.out_cnt = counts;
  if (counts) CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)total * sizeof(int32_t), st));
  for (long long p0 = 0; p0 < total; p0 += batch) {
    a.pair0 = p0;
    a.batch = (int)std::min<long long>(batch, total - p0);
    CUDA_TRY(cudaMemsetAsync(rec, 0, (size_t)a.batch * nb * sizeof(uint4), st));
    CUDA_TRY(launch_large(c, a, st));
  }
  return MFB_OK;
}

// ---------------------------------------------------------------- adjoint
// W_n^m twiddles for the adjoint and the batched four-step: hi[m >> lo_bits] * lo[m & mask],
// built once per (device, n) from FP64 roots.
struct AdjTables {
  float2 *hi = nullptr, *lo = nullptr;   // roots (also the batched launch's)
  float2 *lo_less_one = nullptr;         // lo - 1, the adjoint kernel's
  int lo_bits = 0, hi_count = 0;
};
static std::map<std::pair<int, int>, AdjTables> g_adj;

static int get_adj_tables(int device, int n, AdjTables **out) {
  std::lock_guard<std::mutex> lk(g_const_mu);
  auto it = g_adj.find({device, n});
  if (it != g_adj.end()) { *out = &it->second; return MFB_OK; }
  int L = 0;
  while ((1 << L) < n) L++;
  AdjTables t;
  t.lo_bits = (L + 1) / 2;
  t.hi_count = n >> t.lo_bits;
  std::vector<float2> hi(t.hi_count), lo((size_t)1 << t.lo_bits);
  for (int i = 0; i < t.hi_count; i++) hi[i] = unit_root((long long)i << t.lo_bits, n);
  std::vector<float2> less(lo.size());
  for (size_t i = 0; i < lo.size(); i++) {
    lo[i] = unit_root((long long)i, n);
    // W^i - 1 = 2 i sin(pi i/n) e^(i pi i/n)
    const double s = sin(M_PI * (double)i / n), c = cos(M_PI * (double)i / n);
    less[i] = make_float2((float)(-2.0 * s * s), (float)(2.0 * s * c));
  }
  const size_t lo_bytes = lo.size() * sizeof(float2);
  CUDA_TRY(cudaMalloc(&t.hi, hi.size() * sizeof(float2)));
  CUDA_TRY(cudaMalloc(&t.lo, 2 * lo_bytes));
  t.lo_less_one = t.lo + lo.size();
  CUDA_TRY(cudaMemcpy(t.hi, hi.data(), hi.size() * sizeof(float2), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(t.lo, lo.data(), lo_bytes, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(t.lo_less_one, less.data(), lo_bytes, cudaMemcpyHostToDevice));
  // adjoint_kernel's largest shape (88 KB bounds them all: 40 KB of staged twiddles,
  // 12 of entries, 16 of roots and 16 of list ends)
  CUDA_TRY(cudaFuncSetAttribute(adjoint_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 88 << 10));
  CUDA_TRY(cudaFuncSetAttribute(adjoint_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 88 << 10));
  *out = &(g_adj[{device, n}] = t);
  return MFB_OK;
}

// Dynamic shared memory of adjoint_kernel: the staged twiddles, the sorted
// entries, the twiddle halves and the lists' bucket ends.
static size_t adjoint_smem(int fblk, int items, int roots) {
  const int cap = ADJ_TAB / adj_entry_bytes(fblk);
  return (size_t)ADJ_TAB + (size_t)cap * 12 + 32 + (size_t)roots * 8 + (size_t)items * sizeof(uint4);
}

// One side of the adjoint: a CTA covers 256 (own row, f0) and all other rows;
// when that leaves the device less than ADJ_FILL CTAs per SM, the summed rows
// split over blockIdx.y with atomic accumulation.  A long chain of atomics rounds
// like a long chain of rows, and worse than a balanced split of both, so with
// few tiles (up to ADJ_FEW, where the split is wide) clusters of CTAs add up
// their sums first, in one wave of CTAs that leaves clusters room to be placed
// (7/8 of two per SM); otherwise a CTA sums two rows or more.  B200, gradient of
// 3 rows, 3 x 872 pairs at n = 2048: 291 splits without clusters 33 us and a
// relative error of 3.3e-7, two waves of clusters 42 us and 1.6e-7, this 31.6 us
// and 1.4e-7.
constexpr int ADJ_FILL = 4;
constexpr int ADJ_FEW = 16;
struct AdjPlan {
  int fblk, slots, fx;      // f0 values and own rows per CTA, blocks of f0 values
  long long tiles, split;   // CTAs of one split, splits of the summed rows
  int rows;                 // summed rows per split
  int clusters;
};
static AdjPlan adjoint_plan(int n, int own, int other, int sms) {
  AdjPlan p;
  p.fblk = std::min(n / ADJ_R, ADJ_THREADS);
  p.slots = ADJ_THREADS / p.fblk;
  p.fx = n / ADJ_R / p.fblk;
  p.tiles = (long long)p.fx * ((own + p.slots - 1LL) / p.slots);
  const long long target = (long long)ADJ_FILL * sms;
  p.split = 1;
  if (p.tiles < target) p.split = std::min<long long>(other, target / p.tiles);
  // clusters that fit one wave; a device of few SMs (a partition) may have room for none
  const long long fit = 7LL * sms / 4 / p.tiles / ADJ_CLUSTER * ADJ_CLUSTER;
  p.clusters = p.tiles <= ADJ_FEW && p.split > ADJ_CLUSTER && fit > 0;
  if (p.clusters) p.split = std::min(p.split, fit);
  else if (p.tiles > ADJ_FEW) p.split = std::min<long long>(p.split, std::max(1, other / 2));
  p.rows = (int)((other + p.split - 1) / p.split);
  p.split = (other + p.rows - 1LL) / p.rows;
  if (p.clusters) p.split = (p.split + ADJ_CLUSTER - 1) / ADJ_CLUSTER * ADJ_CLUSTER;   // the last may have no rows
  return p;
}

// adjoint_direct_kernel: own rows per CTA (oc) shrink, and then the summed rows split
// over blockIdx.z, until the grid covers the device about twice; splits past a cluster
// or two are summed by clusters.
struct AdjDirectPlan {
  int oc, fx, chunks, clusters, rows;
  long long split;
};
static AdjDirectPlan adjoint_direct_plan(int n, int own, int other, int sms) {
  AdjDirectPlan p;
  p.fx = ((n >> 1) + ADJ_THREADS - 1) / ADJ_THREADS;
  const long long target = 2LL * sms;
  p.oc = 8;
  while (p.oc > 1 && (long long)p.fx * ((own + p.oc - 1) / p.oc) < target) p.oc >>= 1;
  p.chunks = (own + p.oc - 1) / p.oc;
  const long long tiles = (long long)p.fx * p.chunks;
  p.split = tiles < target ? std::min<long long>(other, (target + tiles - 1) / tiles) : 1;
  p.rows = (int)((other + p.split - 1) / p.split);
  p.split = (other + p.rows - 1LL) / p.rows;
  p.clusters = p.oc == 1 && p.split > ADJD_ATOMICS;
  if (p.clusters) p.split = (p.split + ADJ_CLUSTER - 1) / ADJ_CLUSTER * ADJ_CLUSTER;   // the last may have no rows
  return p;
}

// Whether a gradient takes adjoint_direct_kernel: few entries in all (the limit falls with
// n, whose frequencies the buckets share 16 to a thread), or too few per pair to pay for a
// pair's 16-point transform; not where a CTA would sum more than ADJD_ROWS rows (the
// buckets round less), nor at the longest n with few own rows, where the buckets fill the
// device.  B200, one gradient (own x other rows, bins), us direct against buckets:
// n = 64, 32 x 32 of 4 6.9 / 15.1; n = 1024, 3 x 32 of 16 8.6 / 11.0; n = 4096, 8 x 8 of 4
// 8.3 / 9.7, 128 x 8 of 1 11.8 / 18.9; and past the line n = 1024, 32 x 512 of 16
// 190 / 68, n = 4096, 128 x 8 of 16 48 / 23, n = 262144, 1 x 32 of 1 91 / 24.
static bool adjoint_direct(int n, int own, int other, int nb, int rows) {
  if (rows > ADJD_ROWS || (n > 65536 && own < 4)) return false;
  if (nb == 1 || (n <= 256 && nb <= 4) || (nb == 2 && other <= 2)) return true;
  const double entries = (double)n * own * other * nb;
  const int limit = n <= 256 ? 1 << 25 : n <= 2048 || nb == 2 ? 1 << 23 : 1 << 22;
  return entries <= (other <= 2 ? limit / 2 : limit);
}

extern "C" int mfb_adjoint_plan(size_t n, int own, int other, size_t nb, int sms, int64_t *out) {
  if (!mfb_supported(n) || own < 1 || other < 1 || nb < 1 || nb > n || sms < 1 || !out)
    return fail(MFB_ERR_ARG, "adjoint plan: bad arguments");
  const AdjDirectPlan d = adjoint_direct_plan((int)n, own, other, sms);
  if (adjoint_direct((int)n, own, other, (int)nb, d.rows)) {
    out[0] = (long long)d.fx * d.chunks; out[1] = d.split; out[2] = d.rows; out[3] = d.clusters;
    out[4] = 1;
    return MFB_OK;
  }
  const AdjPlan p = adjoint_plan((int)n, own, other, sms);
  out[0] = p.tiles; out[1] = p.split; out[2] = p.rows; out[3] = p.clusters; out[4] = 0;
  return MFB_OK;
}

// A launch in clusters of ADJ_CLUSTER along the given grid dimension, or without.
template <typename Args>
static cudaError_t launch_adjoint(void (*kernel)(Args), dim3 grid, size_t smem, int cy, int cz,
                                  const Args &a, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = grid;
  cfg.blockDim = dim3(ADJ_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 1;
  attr.val.clusterDim.y = cy;
  attr.val.clusterDim.z = cz;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

template <bool GD>
static int adjoint_direct_side(int n, int nd, int nt, int nb, const float2 *src, const int64_t *idx,
                               const float2 *gz, float2 *out, const AdjTables &tw,
                               const AdjDirectPlan &p, cudaStream_t st) {
  AdjDirectArgs a;
  memset(&a, 0, sizeof a);
  a.src = src; a.idx = idx; a.gz = gz; a.out = out;
  a.n = n; a.nd = nd; a.nt = nt; a.nb = nb;
  a.own = GD ? nd : nt;
  a.other = GD ? nt : nd;
  a.tw_hi = tw.hi; a.tw_lo = tw.lo; a.lo_bits = tw.lo_bits; a.hi_count = tw.hi_count;
  a.other_per_split = p.rows; a.accumulate = p.split > 1; a.clusters = p.clusters;
  a.bins_per_round = std::min(nb, ADJD_CAP / p.oc);
  a.rows_per_round = a.bins_per_round == nb ? ADJD_CAP / (p.oc * nb) : 1;
  if (a.accumulate) CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)a.own * n * sizeof(float2), st));
  const dim3 grid((unsigned)p.fx, (unsigned)p.chunks, (unsigned)p.split);
  auto kernel = p.oc == 8   ? adjoint_direct_kernel<8, GD>
                : p.oc == 4 ? adjoint_direct_kernel<4, GD>
                : p.oc == 2 ? adjoint_direct_kernel<2, GD>
                            : adjoint_direct_kernel<1, GD>;
  CUDA_TRY(launch_adjoint(kernel, grid, 0, 1, p.clusters ? ADJ_CLUSTER : 1, a, st));
  return MFB_OK;
}

static int adjoint_side(bool grad_data, int n, int nd, int nt, int nb, const float2 *src,
                        const int64_t *idx, const float2 *gz, float2 *out, const AdjTables &tw,
                        int sms, cudaStream_t st) {
  AdjArgs a;
  memset(&a, 0, sizeof a);
  a.src = src; a.idx = idx; a.gz = gz; a.out = out;
  a.n = n; a.nd = nd; a.nt = nt; a.nb = nb;
  a.own = grad_data ? nd : nt;
  a.other = grad_data ? nt : nd;
  if ((a.own + 7LL) / 8 > 65535) return fail(MFB_ERR_UNSUPPORTED, "adjoint: too many rows (%d)", a.own);
  const AdjDirectPlan dp = adjoint_direct_plan(n, a.own, a.other, sms);
  if (adjoint_direct(n, a.own, a.other, nb, dp.rows))
    return grad_data ? adjoint_direct_side<true>(n, nd, nt, nb, src, idx, gz, out, tw, dp, st)
                     : adjoint_direct_side<false>(n, nd, nt, nb, src, idx, gz, out, tw, dp, st);
  const AdjPlan p = adjoint_plan(n, a.own, a.other, sms);
  a.fblk = p.fblk; a.slots = p.slots; a.fx = p.fx;
  a.other_per_split = p.rows; a.clusters = p.clusters; a.accumulate = p.split > 1;
  while ((1 << a.lsh) < a.fblk && a.lsh < 5) a.lsh++;
  while ((32 << a.ash) < a.fblk) a.ash++;
  a.tw_hi = tw.hi; a.tw_lo = tw.lo_less_one; a.lo_bits = tw.lo_bits; a.hi_count = tw.hi_count;
  const int cap = ADJ_TAB / adj_entry_bytes(a.fblk);
  a.chunk = std::min(std::min(nb, ADJ_CHUNK), cap / a.slots);
  a.chunks = (nb + a.chunk - 1) / a.chunk;
  const int lists = std::min(cap / (a.chunk * a.slots), ADJ_ITEMS / a.slots);   // per own row and round
  a.rows_per_round = a.chunks == 1 ? lists : 1;
  a.lists_per_round = a.chunks == 1 ? 1 : std::min(lists, a.chunks);
  if (a.accumulate) CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)a.own * n * sizeof(float2), st));
  const dim3 grid((unsigned)p.tiles, (unsigned)p.split);
  const size_t smem = adjoint_smem(a.fblk, lists * a.slots, tw.hi_count + (1 << tw.lo_bits));
  CUDA_TRY(launch_adjoint(grad_data ? adjoint_kernel<true> : adjoint_kernel<false>, grid, smem,
                          a.clusters ? ADJ_CLUSTER : 1, 1, a, st));
  return MFB_OK;
}

extern "C" int mfb_adjoint(int device, size_t n, const void *data, int nd, const void *templates,
                           int nt, size_t nb, const int64_t *idx, const void *gz, void *grad_data,
                           void *grad_tmpl, void *stream) {
  if (!mfb_supported(n)) return fail(MFB_ERR_UNSUPPORTED, "adjoint: unsupported n=%zu", n);
  if (nd < 1 || nt < 1 || nb < 1 || nb > n) return fail(MFB_ERR_ARG, "adjoint: bad shape");
  if (!data || !templates || !idx || !gz) return fail(MFB_ERR_ARG, "adjoint: null input");
  int ndev = 0;
  CUDA_TRY(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev) return fail(MFB_ERR_ARG, "no device %d", device);
  DeviceGuard dg(device);
  AdjTables *tw = nullptr;
  int r = get_adj_tables(device, (int)n, &tw);
  if (r) return r;
  int sms = 0;
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  cudaStream_t st = (cudaStream_t)stream;
  if (grad_data) {
    r = adjoint_side(true, (int)n, nd, nt, (int)nb, (const float2 *)templates, idx,
                     (const float2 *)gz, (float2 *)grad_data, *tw, sms, st);
    if (r) return r;
  }
  if (grad_tmpl) {
    r = adjoint_side(false, (int)n, nd, nt, (int)nb, (const float2 *)data, idx,
                     (const float2 *)gz, (float2 *)grad_tmpl, *tw, sms, st);
    if (r) return r;
  }
  return MFB_OK;
}

// ---------------------------------------------------------------- batched jobs
struct mfb_batch {
  int device = 0;
  BatchArgs args;
  void *arena = nullptr;          // jobs, segments, batch totals, counters
  void *table = nullptr;          // device copy of the constant table (args + jobs)
  size_t table_bytes = 0;
  void *counters = nullptr;       // ticket, a_done, b_done, fwd_done, err: cleared every run
  size_t counter_bytes = 0;
  std::vector<std::pair<void *, size_t>> rec_clear;   // two-pass outputs, cleared every run
  std::vector<void *> owned;      // series workspaces and block starts
  float2 *slots = nullptr;
  int grid = 0, smem = 0, nbatch = 0;
  size_t scratch_bytes = 0;
};

static void batch_free(mfb_batch *b) {
  if (!b) return;
  DeviceGuard dg(b->device);
  cudaFree(b->arena);
  cudaFree(b->slots);
  for (void *p : b->owned) cudaFree(p);
  delete b;
}

extern "C" int mfb_batch_destroy(mfb_batch *b) {
  batch_free(b);
  return MFB_OK;
}

namespace {
struct PendingBatch { int job, q_local, count; };
}

extern "C" int mfb_batch_create(mfb_batch **out, int device, const mfb_job *jobs, int njobs,
                                const mfb_batch_opts *opts) {
  if (!out) return fail(MFB_ERR_ARG, "null output handle");
  *out = nullptr;
  if (!jobs || njobs < 1) return fail(MFB_ERR_ARG, "no jobs");
  if (njobs > BATCH_MAX_JOBS)
    return fail(MFB_ERR_UNSUPPORTED, "%d jobs; one batch takes at most %d", njobs, BATCH_MAX_JOBS);
  int ndev = 0;
  CUDA_TRY(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev) return fail(MFB_ERR_ARG, "no device %d", device);
  const size_t slot_bytes = (opts && opts->slot_bytes) ? opts->slot_bytes : ((size_t)64 << 20);
  const int nslots = (opts && opts->slots) ? opts->slots : 3;
  if (nslots < 2 || nslots > 64) return fail(MFB_ERR_ARG, "slots must be 2 .. 64");
  DeviceGuard dg(device);
  std::unique_ptr<mfb_batch, void (*)(mfb_batch *)> b(new mfb_batch, batch_free);
  b->device = device;
  memset(&b->args, 0, sizeof b->args);
  std::vector<BatchJob> hj(njobs);
  bool any_two = false;
  for (int i = 0; i < njobs; i++) {
    const mfb_job &J = jobs[i];
    BatchJob &j = hj[i];
    memset(&j, 0, sizeof j);
    const size_t n = J.n;
    if (!mfb_supported(n)) return fail(MFB_ERR_UNSUPPORTED, "job %d: unsupported n=%zu", i, n);
    if (J.nd < 1 || J.nt < 1) return fail(MFB_ERR_ARG, "job %d: nd and nt must be >= 1", i);
    if (!J.templates || !J.records) return fail(MFB_ERR_ARG, "job %d: null templates or records", i);
    if (((uintptr_t)J.records & 15u) != 0) return fail(MFB_ERR_ARG, "job %d: records not 16-byte aligned", i);
    const bool series = J.series != nullptr;
    if (series ? (!J.starts || J.nseries < 1) : !J.data)
      return fail(MFB_ERR_ARG, "job %d: give data spectra, or series with block starts", i);
    if (J.binsize < 1) return fail(MFB_ERR_ARG, "job %d: binsize must be >= 1", i);
    if (std::isnan(J.threshold)) return fail(MFB_ERR_ARG, "job %d: threshold is NaN", i);
    const size_t nb = mfb_nbins(n, J.binsize, J.start, J.end);
    if (nb == 0) return fail(MFB_ERR_ARG, "job %d: empty window [%zu, %zu)", i, J.start, J.end);
    j.n = (int)n; j.nd = J.nd; j.nt = J.nt; j.nb = (int)nb;
    j.binsize = J.binsize > n ? (int)n : (int)J.binsize;
    j.ws = (int)J.start;
    j.we = (int)(J.end > n ? n : J.end);
    j.t2 = J.threshold > 0.f ? J.threshold * J.threshold : 0.f;
    j.tmpl = (const float2 *)J.templates;
    j.rec = (uint4 *)J.records;
    j.scale = 1.0f / (float)n;
    j.fwd_ctr = i;
    int L = 0;
    while (((size_t)1 << L) < n) L++;
    if (n <= 4096) {
      NConst *c = nullptr;
      int r = get_const(device, (int)n, &c);
      if (r) return r;
      j.twid = c->twid;
      j.unit_items = J.unit_items > 0 ? J.unit_items : 1;
    } else {
      any_two = true;
      const int N2 = J.split ? J.split : (n >= 16384 ? 256 : 128);
      if (N2 != 64 && N2 != 128 && N2 != 256)
        return fail(MFB_ERR_ARG, "job %d: split (N2) must be 64, 128 or 256", i);
      const size_t N1 = n / (size_t)N2;
      if (N1 < 64 || N1 > 4096)
        return fail(MFB_ERR_UNSUPPORTED, "job %d: n=%zu with N2=%d gives N1=%zu outside 64 .. 4096",
                    i, n, N2, N1);
      if (nb > (size_t)BATCH_MAX_BINS)
        return fail(MFB_ERR_UNSUPPORTED, "job %d: %zu bins per pair; n >= 8192 takes at most %d", i,
                    nb, BATCH_MAX_BINS);
      if (n * sizeof(float2) > slot_bytes)
        return fail(MFB_ERR_ARG, "job %d: one pair (%zu bytes) does not fit a %zu-byte slot", i,
                    n * sizeof(float2), slot_bytes);
      j.N1 = (int)N1; j.N2 = N2;
      NConst *c1 = nullptr, *c2 = nullptr;
      AdjTables *tw = nullptr;
      int r = get_const(device, (int)N1, &c1);
      if (!r) r = get_const(device, N2, &c2);
      if (!r) r = get_adj_tables(device, (int)n, &tw);
      if (r) return r;
      j.tw1 = c1->twid; j.tw2 = c2->twid;
      j.tw_hi = tw->hi; j.tw_lo = tw->lo; j.lo_bits = tw->lo_bits;
      j.batch_pairs = (int)std::max<size_t>(1, slot_bytes / (n * sizeof(float2)));
      b->rec_clear.push_back({J.records, (size_t)J.nd * J.nt * nb * 16});
    }
    if (series) {
      void *spec = nullptr, *st = nullptr;
      CUDA_TRY(cudaMalloc(&spec, (size_t)J.nd * n * sizeof(float2)));
      b->owned.push_back(spec);
      CUDA_TRY(cudaMalloc(&st, (size_t)J.nd * sizeof(uint64_t)));
      b->owned.push_back(st);
      CUDA_TRY(cudaMemcpy(st, J.starts, (size_t)J.nd * sizeof(uint64_t), cudaMemcpyHostToDevice));
      j.spec = (float2 *)spec;
      j.data = (const float2 *)spec;
      j.series = (const float2 *)J.series;
      j.nseries = (long long)J.nseries;
      j.starts = (const unsigned long long *)st;
    } else {
      j.data = (const float2 *)J.data;
    }
  }

  // Segments: forward transforms first, then the two-pass pipeline, then the
  // single-CTA jobs (largest n first), so every wait is on earlier tickets.
  std::vector<BatchSeg> segs;
  std::vector<unsigned> a_total, b_total;
  long long t = 0;
  // Grid first: A/B tickets take several work units when a segment has
  // enough of them to keep every CTA busy for two tickets.
  const int smem = batch_smem_bytes();
  CUDA_TRY(cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int per_sm = 0, sms = 0;
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel, BATCH_CTA, smem));
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  if (per_sm < 1) return fail(MFB_ERR_CUDA, "batched kernel cannot be resident");
  const long long grid = (long long)per_sm * sms;
  auto add = [&](int job, int kind, int q, int q_local, long long units, int pairs) -> int {
    if (units < 1) return MFB_OK;
    if (units > INT32_MAX) return fail(MFB_ERR_UNSUPPORTED, "job %d: too many units", job);
    BatchSeg s;
    memset(&s, 0, sizeof s);
    s.t0 = t; s.job = job; s.kind = kind; s.q = q; s.q_local = q_local;
    s.pairs = pairs;
    s.raw = (int)units;
    s.per = 1;
    if (kind != SEG_SMALL && kind != SEG_FWD_SMALL)
      s.per = (int)std::max<long long>(1, std::min<long long>(8, units / (2 * grid)));
    s.units = (int)((units + s.per - 1) / s.per);
    segs.push_back(s);
    t += s.units;
    return MFB_OK;
  };
  for (int i = 0; i < njobs; i++) {
    BatchJob &j = hj[i];
    if (j.spec && j.n <= 4096) {
      const int G = 4096 / j.n;
      j.fwd_units = (j.nd + G - 1) / G;
      int r = add(i, SEG_FWD_SMALL, 0, 0, j.fwd_units, 0);
      if (r) return r;
    }
  }
  int q = 0;
  auto pipeline = [&](const std::vector<PendingBatch> &list, int kind_a, int kind_b) -> int {
    const int q0 = q;
    for (size_t k = 0; k < list.size(); k++) {
      const BatchJob &j = hj[list[k].job];
      const unsigned units = (unsigned)((long long)list[k].count * (j.n / 4096));
      a_total.push_back(units);
      b_total.push_back(units);
      q++;
    }
    for (size_t k = 0; k <= list.size(); k++) {
      if (k < list.size()) {
        const PendingBatch &p = list[k];
        int r = add(p.job, kind_a, q0 + (int)k, p.q_local, a_total[q0 + k], p.count);
        if (r) return r;
      }
      if (k >= 1) {
        const PendingBatch &p = list[k - 1];
        int r = add(p.job, kind_b, q0 + (int)k - 1, p.q_local, b_total[q0 + k - 1], p.count);
        if (r) return r;
      }
    }
    return MFB_OK;
  };
  std::vector<PendingBatch> fwd_list, pair_list;
  for (int i = 0; i < njobs; i++) {
    BatchJob &j = hj[i];
    if (j.n <= 4096) continue;
    if (j.spec) {
      for (int q_local = 0, b0 = 0; b0 < j.nd; q_local++, b0 += j.batch_pairs) {
        const int c = std::min(j.batch_pairs, j.nd - b0);
        fwd_list.push_back({i, q_local, c});
        j.fwd_units += c * (j.n / 4096);
      }
    }
    const long long pairs = (long long)j.nd * j.nt;
    long long q_local = 0;
    for (long long p0 = 0; p0 < pairs; p0 += j.batch_pairs, q_local++) {
      if (q_local > INT32_MAX) return fail(MFB_ERR_UNSUPPORTED, "job %d: too many batches", i);
      pair_list.push_back({i, (int)q_local, (int)std::min<long long>(j.batch_pairs, pairs - p0)});
    }
  }
  int r = pipeline(fwd_list, SEG_FA, SEG_FB);
  if (!r) r = pipeline(pair_list, SEG_A, SEG_B);
  if (r) return r;
  std::vector<int> small;
  for (int i = 0; i < njobs; i++)
    if (hj[i].n <= 4096) small.push_back(i);
  std::stable_sort(small.begin(), small.end(), [&](int x, int y) { return hj[x].n > hj[y].n; });
  for (int i : small) {
    const BatchJob &j = hj[i];
    const long long G = 4096 / j.n;
    const long long items = ((long long)j.nd * j.nt + G - 1) / G;
    r = add(i, SEG_SMALL, 0, 0, (items + j.unit_items - 1) / j.unit_items, 0);
    if (r) return r;
  }
  if (segs.empty()) return fail(MFB_ERR_ARG, "no work");

  // One arena: table (args + jobs) | segments | a_total | b_total | counters.
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const int Q = (int)a_total.size();
  b->table_bytes = offsetof(BatchTable, jobs) + njobs * sizeof(BatchJob);
  const size_t o_jobs = 0, o_segs = up(b->table_bytes);
  const size_t o_at = o_segs + up(segs.size() * sizeof(BatchSeg));
  const size_t o_bt = o_at + up(Q * sizeof(unsigned) + 4);
  const size_t o_ctr = o_bt + up(Q * sizeof(unsigned) + 4);
  const size_t ctr_bytes = 8 + 2 * (size_t)Q * sizeof(unsigned) + (size_t)njobs * sizeof(unsigned) + 8;
  CUDA_TRY(cudaMalloc(&b->arena, o_ctr + up(ctr_bytes)));
  char *base = (char *)b->arena;
  b->table = base + o_jobs;
  CUDA_TRY(cudaMemcpy(base + o_segs, segs.data(), segs.size() * sizeof(BatchSeg),
                      cudaMemcpyHostToDevice));
  if (Q) {
    CUDA_TRY(cudaMemcpy(base + o_at, a_total.data(), Q * sizeof(unsigned), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(base + o_bt, b_total.data(), Q * sizeof(unsigned), cudaMemcpyHostToDevice));
  }
  char *ctr = base + o_ctr;
  b->counters = ctr;
  b->counter_bytes = ctr_bytes;
  BatchArgs &A = b->args;
  A.segs = (const BatchSeg *)(base + o_segs);
  A.nseg = (int)segs.size();
  A.total = t;
  A.ticket = (unsigned long long *)ctr;
  A.a_done = (unsigned *)(ctr + 8);
  A.b_done = A.a_done + Q;
  A.fwd_done = A.b_done + Q;
  A.err = (int *)(A.fwd_done + njobs);
  A.a_total = (const unsigned *)(base + o_at);
  A.b_total = (const unsigned *)(base + o_bt);
  A.nslots = nslots;
  A.slot_elems = (long long)(slot_bytes / sizeof(float2));
  if (any_two) {
    CUDA_TRY(cudaMalloc(&b->slots, (size_t)nslots * slot_bytes));
    b->scratch_bytes = (size_t)nslots * slot_bytes;
  }
  A.slots = b->slots;
  b->nbatch = Q;
  {
    std::vector<char> table(b->table_bytes);
    memcpy(table.data() + offsetof(BatchTable, args), &A, sizeof A);
    memcpy(table.data() + offsetof(BatchTable, jobs), hj.data(), njobs * sizeof(BatchJob));
    CUDA_TRY(cudaMemcpy(b->table, table.data(), b->table_bytes, cudaMemcpyHostToDevice));
  }
  b->smem = smem;
  b->grid = (int)grid;
  *out = b.release();
  return MFB_OK;
}

extern "C" int mfb_batch_run(mfb_batch *b, void *stream) {
  if (!b) return fail(MFB_ERR_ARG, "null batch");
  DeviceGuard dg(b->device);
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(cudaMemcpyToSymbolAsync(c_batch, b->table, b->table_bytes, 0,
                                    cudaMemcpyDeviceToDevice, st));
  CUDA_TRY(cudaMemsetAsync(b->counters, 0, b->counter_bytes, st));
  for (auto &z : b->rec_clear) CUDA_TRY(cudaMemsetAsync(z.first, 0, z.second, st));
  batch_kernel<<<b->grid, BATCH_CTA, b->smem, st>>>();
  CUDA_TRY(cudaGetLastError());
  return MFB_OK;
}

extern "C" int mfb_batch_status(mfb_batch *b, void *stream) {
  if (!b) return fail(MFB_ERR_ARG, "null batch");
  DeviceGuard dg(b->device);
  CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  int err = 0;
  CUDA_TRY(cudaMemcpy(&err, b->args.err, sizeof err, cudaMemcpyDeviceToHost));
  if (err) return fail(MFB_ERR_CUDA, "batched launch stopped: a dependency wait ran out (code %d)", err);
  return MFB_OK;
}

extern "C" int mfb_batch_test_wait_limit(mfb_batch *b, int delta) {
  if (!b) return fail(MFB_ERR_ARG, "null batch");
  if (b->nbatch < 1 || !b->args.a_total)
    return fail(MFB_ERR_STATE, "the batch has no four-step pass to hold back");
  if (delta != 1 && delta != -1) return fail(MFB_ERR_ARG, "delta must be +1 or -1");
  DeviceGuard dg(b->device);
  CUDA_TRY(cudaDeviceSynchronize());
  unsigned *at = const_cast<unsigned *>(b->args.a_total);
  unsigned v = 0;
  CUDA_TRY(cudaMemcpy(&v, at, sizeof v, cudaMemcpyDeviceToHost));
  v += (unsigned)delta;
  CUDA_TRY(cudaMemcpy(at, &v, sizeof v, cudaMemcpyHostToDevice));
  return MFB_OK;
}

extern "C" int mfb_batch_info(mfb_batch *b, int64_t *tickets, int *grid, int *segments,
                              int *batches, size_t *scratch_bytes) {
  if (!b) return fail(MFB_ERR_ARG, "null batch");
  if (tickets) *tickets = b->args.total;
  if (grid) *grid = b->grid;
  if (segments) *segments = b->args.nseg;
  if (batches) *batches = b->nbatch;
  if (scratch_bytes) *scratch_bytes = b->scratch_bytes;
  return MFB_OK;
}

// ------------------------------------------------- hierarchical run_series
static int hier_run_series_impl(mfb_hplan *h, const void *series, size_t nseries,
                                const uint64_t *starts, const uint64_t *win_start,
                                const uint64_t *win_end, int nblocks, int t0, int nt,
                                size_t binsize, float threshold, int64_t *idx, void *val,
                                int32_t *counts, int rs) {
  if (!h) return fail(MFB_ERR_ARG, "null plan");
  mfb_plan *p = h->full;
  if (!series || !starts || !win_start || !win_end || nblocks < 1 || !idx || !val)
    return fail(MFB_ERR_ARG, "invalid run_series arguments");
  if (t0 < 0 || nt < 1 || t0 > p->nt - nt || binsize < 1)
    return fail(MFB_ERR_ARG, "invalid template range or binsize");
  size_t nb0 = 0;
  for (int b = 0; b < nblocks; b++) {   // equal bin counts (src/hmf.c:199-213)
    size_t lo = win_start[b], hi = win_end[b] > p->n ? p->n : win_end[b];
    if (lo >= hi || starts[b] > (uint64_t)INT64_MAX - p->n)
      return fail(MFB_ERR_ARG, "block %d has an empty window or an overflowing start", b);
    size_t nb = 1 + (hi - lo - 1) / binsize;
    if (b == 0) nb0 = nb;
    else if (nb != nb0) return fail(MFB_ERR_ARG, "block windows must have equal bin counts");
  }
  DeviceGuard dg(h->device);
  if (p->starts_cap < nblocks) {
    cudaFree(p->starts_dev);
    p->starts_dev = nullptr;
    p->starts_cap = 0;
    CUDA_TRY(cudaMalloc(&p->starts_dev, (size_t)nblocks * sizeof(uint64_t)));
    p->starts_cap = nblocks;
  }
  CUDA_TRY(cudaMemcpyAsync(p->starts_dev, starts, (size_t)nblocks * sizeof(uint64_t),
                           cudaMemcpyHostToDevice, p->stream));
  // Runs of equal windows, at most ndata blocks each, transformed straight into
  // the plan's data rows (src/hmf.c:171-197) and filtered hierarchically.
  for (int b0 = 0; b0 < nblocks;) {
    int g = 1;
    while (g < p->nd && b0 + g < nblocks && win_start[b0 + g] == win_start[b0] &&
           win_end[b0 + g] == win_end[b0])
      g++;
    int r = mfb_forward(p, series, nseries, p->starts_dev + b0, g, p->data);
    if (r) return r;
    r = hier_run_impl(h, 0, g, t0, nt, binsize, threshold, win_start[b0], win_end[b0],
                      idx + (size_t)b0 * nt * nb0 * rs, (float2 *)val + (size_t)b0 * nt * nb0 * rs,
                      counts ? counts + (size_t)b0 * nt : nullptr, rs);
    if (r) return r;
    b0 += g;
  }
  return MFB_OK;
}
extern "C" int mfb_hier_run_series(mfb_hplan *h, const void *series, size_t nseries,
                                   const uint64_t *starts, const uint64_t *win_start,
                                   const uint64_t *win_end, int nblocks, int t0, int nt,
                                   size_t binsize, float threshold, int64_t *idx, void *val,
                                   int32_t *counts) {
  return hier_run_series_impl(h, series, nseries, starts, win_start, win_end, nblocks, t0, nt, binsize,
                              threshold, idx, val, counts, 1);
}
extern "C" int mfb_hier_run_series_records(mfb_hplan *h, const void *series, size_t nseries,
                                           const uint64_t *starts, const uint64_t *win_start,
                                           const uint64_t *win_end, int nblocks, int t0, int nt,
                                           size_t binsize, float threshold, void *records,
                                           int32_t *counts) {
  if (!records) return fail(MFB_ERR_ARG, "null pointer argument");
  return hier_run_series_impl(h, series, nseries, starts, win_start, win_end, nblocks, t0, nt, binsize,
                              threshold, (int64_t *)records, (char *)records + 8, counts, 2);
}

// --------------------------------------------------------- gate model (device)
extern "C" int mfb_gate_maxima(int device, const double *power, size_t n, size_t band, float snr,
                               int step, int per, int has_out, const int32_t *taus,
                               const int32_t *ntaus, const int32_t *on_grid, const void *draw_in,
                               const void *draw_out, float *coarse, float *fine,
                               double *sums_out) {
  if (!power || !taus || !ntaus || !on_grid || !draw_in || !coarse || !fine)
    return fail(MFB_ERR_ARG, "gate model: null pointer");
  if (n < 64 || n > ((size_t)1 << 20) || band < 1 || band > n || n % band)
    return fail(MFB_ERR_ARG, "gate model: band must divide n (n <= 2^20)");
  if (step != (int)(n / band) || per < 1 || (has_out && !draw_out))
    return fail(MFB_ERR_ARG, "gate model: bad step, per or out-of-band draws");
  if (!std::isfinite(snr) || snr <= 0.f) return fail(MFB_ERR_ARG, "gate model: bad snr");
  const int dmax = 8 * step + 8;
  for (int o = 0; o < step; o++) {
    const int K = ntaus[o];
    if (K < 1 || K > GATE_K) return fail(MFB_ERR_ARG, "gate model: %d lags at offset %d", K, o);
    for (int i = 0; i < K; i++) {
      const int t = taus[o * GATE_K + i];
      if (t < -dmax / 2 || t > dmax / 2 || t - o < -dmax || t - o > dmax)
        return fail(MFB_ERR_ARG, "gate model: lag %d outside the table", t);
    }
    for (int g = 0; g < GATE_GRID; g++)
      if (on_grid[o * GATE_GRID + g] < 0 || on_grid[o * GATE_GRID + g] >= K)
        return fail(MFB_ERR_ARG, "gate model: grid index out of range");
  }
  int ndev = 0;
  CUDA_TRY(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev) return fail(MFB_ERR_ARG, "no device %d", device);
  DeviceGuard dg(device);
  const size_t nl = 2 * (size_t)dmax + 1, kk = (size_t)GATE_K * GATE_K;
  const size_t draws = (size_t)step * per * GATE_K * sizeof(float2);
  const size_t bytes[] = {n * sizeof(double), 2 * sizeof(double), nl * sizeof(double2),
                          nl * sizeof(double2), (size_t)step * GATE_K * sizeof(int),
                          (size_t)step * sizeof(int), (size_t)step * GATE_GRID * sizeof(int),
                          step * kk * sizeof(float2), step * kk * sizeof(float2),
                          (size_t)step * GATE_K * sizeof(float2), (size_t)step * GATE_K * sizeof(float2),
                          draws, has_out ? draws : 0, (size_t)step * per * sizeof(float),
                          (size_t)step * per * sizeof(float)};
  constexpr int NB = sizeof(bytes) / sizeof(bytes[0]);
  size_t off[NB + 1];
  off[0] = 0;
  for (int i = 0; i < NB; i++) off[i + 1] = off[i] + ((bytes[i] + 255) & ~(size_t)255);
  char *mem = nullptr;
  CUDA_TRY(cudaMalloc(&mem, off[NB]));
  std::unique_ptr<char, cudaError_t (*)(void *)> guard(mem, cudaFree);
  GateArgs a;
  memset(&a, 0, sizeof a);
  a.power = (const double *)(mem + off[0]);
  a.sums = (double *)(mem + off[1]);
  a.a_full = (double2 *)(mem + off[2]);
  a.a_band = (double2 *)(mem + off[3]);
  a.taus = (const int *)(mem + off[4]);
  a.ntaus = (const int *)(mem + off[5]);
  a.on_grid = (const int *)(mem + off[6]);
  a.l_in = (float2 *)(mem + off[7]);
  a.l_out = (float2 *)(mem + off[8]);
  a.s_full = (float2 *)(mem + off[9]);
  a.s_band = (float2 *)(mem + off[10]);
  a.draw_in = (const float2 *)(mem + off[11]);
  a.draw_out = has_out ? (const float2 *)(mem + off[12]) : nullptr;
  a.coarse = (float *)(mem + off[13]);
  a.fine = (float *)(mem + off[14]);
  a.n = (int)n; a.band = (int)band; a.dmax = dmax;
  a.step = step; a.per = per; a.has_out = has_out; a.snr = snr;
  CUDA_TRY(cudaMemcpy(mem + off[0], power, bytes[0], cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(mem + off[4], taus, bytes[4], cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(mem + off[5], ntaus, bytes[5], cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(mem + off[6], on_grid, bytes[6], cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(mem + off[11], draw_in, draws, cudaMemcpyHostToDevice));
  if (has_out) CUDA_TRY(cudaMemcpy(mem + off[12], draw_out, draws, cudaMemcpyHostToDevice));
  gate_sums_kernel<<<1, 1024>>>(a);
  CUDA_TRY(cudaGetLastError());
  gate_lags_kernel<<<(unsigned)nl, 256>>>(a);
  CUDA_TRY(cudaGetLastError());
  gate_chol_kernel<<<(step + 63) / 64, 64>>>(a);
  CUDA_TRY(cudaGetLastError());
  gate_draw_kernel<<<dim3((unsigned)((per + 127) / 128), (unsigned)step), 128>>>(a);
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaMemcpy(coarse, a.coarse, bytes[13], cudaMemcpyDeviceToHost));
  CUDA_TRY(cudaMemcpy(fine, a.fine, bytes[14], cudaMemcpyDeviceToHost));
  if (sums_out) CUDA_TRY(cudaMemcpy(sums_out, a.sums, 2 * sizeof(double), cudaMemcpyDeviceToHost));
  return MFB_OK;
}
