// Device-side `naja validate` metrics: Geyer ESS per (dim, chain) and
// split-R-hat per dim, following src/validate/mcmc.cpp:17-194 of
// quothbonney/naja.
//
// ESS: one CTA per series.  The series is centred in shared memory and its
// autocovariances are summed directly (FP32 products, FP64 sums) in blocks of
// lags until Geyer's initial positive sequence stops.  The reference obtains
// the same acov[k] = (1/n) sum (x_t-m)(x_{t+k}-m) from a float FFT of size 2n;
// the direct sum needs only the lags the rule reaches (a few blocks for a
// mixing chain) and has no FFT round-off.
//
// R-hat: half-chain sums in FP64 as mcmc.cpp takes them, eight coordinates (a
// sector of the sample rows) per CTA.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/naja_chr.h"
#include "capi_internal.cuh"

namespace naja {
namespace {

constexpr int kEssThreads = 256;
constexpr long kEssMaxSeries = 48 * 1024;  // floats kept on chip per series

__device__ __forceinline__ long series_row(int layout, int c, long i, long spc, int nchains) {
  return layout == 0 ? static_cast<long>(c) * spc + i : i * nchains + c;
}

__device__ double block_sum(double v, double* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) scratch[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = (l < static_cast<int>(blockDim.x >> 5)) ? scratch[l] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (l == 0) scratch[0] = t;
  }
  __syncthreads();
  t = scratch[0];
  __syncthreads();
  return t;
}

// Lags per thread: a sliding window, one new value per sample for kEssLags
// products.  A block of lags is 4 L of them for L lanes of lags; the threads
// share out the samples in 256 / L slices.
constexpr int kEssLags = 4;
constexpr int kEssMaxBlock = 512;
constexpr int kEssPad = 2 * kEssLags;  // zeros behind a series: a product past its end is 0

// Lags of the block that starts at lag `base`: a mixing chain stops within
// the first few short ones; a block grows with the lags already taken, so that
// the products past the stop and the rounds of barriers both stay a small
// share (700 x 16 series of 2,500 samples, correlation 0.999: 5.5 ms with 64
// lags throughout, 3.9 ms so; 0.98: 2.3 and 1.5 ms).
__device__ __forceinline__ int ess_block(long base) {
  return base <= 256 ? 64 : base <= 512 ? 128 : base <= 1536 ? 256 : kEssMaxBlock;
}

// One CTA per series.  What bounds it is the conversion of each FP32 product
// to FP64 (16 per clock and SM), so the gain is in the products not taken:
// first blocks of 64 lags instead of 512, and a stopping rule that takes a
// block's pairs side by side.  Eight series per CTA, one after another, read
// whole sectors of the rows but left SMs idle where there are few series
// (50 x 2 of 2,500, correlation 0.98: 469 us, 81 one by one), and with many
// the loads are no bound.
__global__ void __launch_bounds__(kEssThreads) ess_kernel(const float* __restrict__ s, long N, int dim, int nchains,
                                                        int layout, double* __restrict__ ess) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ double scratch[32];
  __shared__ __align__(16) double part_lag[kEssThreads * kEssLags];  // [slice][lag]
  __shared__ double pairs[kEssMaxBlock / 2];
  __shared__ int first_negative;
  __shared__ double tau_sh;
  float* y = reinterpret_cast<float*>(sm);
  const long n = N / nchains, series = blockIdx.x;
  const int c = blockIdx.x % nchains;
  {
    const float* src = s + series_row(layout, c, 0, n, nchains) * dim + blockIdx.x / nchains;
    const long step = static_cast<long>(layout == 0 ? 1 : nchains) * dim;
    for (int i = threadIdx.x; i < n + kEssPad; i += kEssThreads) y[i] = i < n ? src[i * step] : 0.0f;
  }
  __syncthreads();
  double part = 0.0;
  for (long i = threadIdx.x; i < n; i += kEssThreads) part += static_cast<double>(y[i]);
  const double mean = block_sum(part, scratch) / static_cast<double>(n);
  part = 0.0;
  for (long i = threadIdx.x; i < n; i += kEssThreads) {
    const float v = static_cast<float>(static_cast<double>(y[i]) - mean);
    y[i] = v;
    part += static_cast<double>(v) * v;
  }
  const double var = block_sum(part, scratch) / static_cast<double>(n);  // acov[0]
  if (var < 1e-30) {
    if (threadIdx.x == 0) ess[series] = 1.0;
    return;
  }
  if (threadIdx.x == 0) {
    first_negative = kEssMaxBlock;
    tau_sh = 1.0;
  }
  // pair k uses lags 2k-1, 2k, for k = 1 .. kmax-1
  const long kmax = n / 2;
  int block;
  for (long base = 1; base <= 2 * (kmax - 1); base += block) {
    block = ess_block(base);
    const int lanes = block / kEssLags, slices = kEssThreads / lanes;
    const int li = threadIdx.x & (lanes - 1), slice = threadIdx.x / lanes;
    // this thread: lags lag0 .. lag0 + 3 over its slice of t < n - lag0
    // (beyond that every product is 0)
    const long lag0 = base + li * kEssLags;
    double acc[kEssLags];
#pragma unroll
    for (int j = 0; j < kEssLags; ++j) acc[j] = 0.0;
    if (lag0 < n) {
      const int len = static_cast<int>(n - lag0);
      const int t0 = static_cast<int>(static_cast<long>(len) * slice / slices);
      const int t1 = static_cast<int>(static_cast<long>(len) * (slice + 1) / slices);
      const float* yk = y + lag0;
      float w[kEssLags];
#pragma unroll
      for (int j = 0; j < kEssLags; ++j) w[j] = yk[t0 + j];
      int t = t0;
#pragma unroll 4
      for (; t + kEssLags <= t1; t += kEssLags) {
        float next[kEssLags];
#pragma unroll
        for (int j = 0; j < kEssLags; ++j) next[j] = yk[t + kEssLags + j];
#pragma unroll
        for (int u = 0; u < kEssLags; ++u) {
          const float v = y[t + u];
#pragma unroll
          for (int j = 0; j < kEssLags; ++j)
            acc[j] += static_cast<double>(v * (u + j < kEssLags ? w[(u + j) % kEssLags] : next[(u + j) % kEssLags]));
        }
#pragma unroll
        for (int j = 0; j < kEssLags; ++j) w[j] = next[j];
      }
      for (; t < t1; ++t) {
        const float v = y[t];
#pragma unroll
        for (int j = 0; j < kEssLags; ++j) acc[j] += static_cast<double>(v * yk[t + j]);
      }
    }
#pragma unroll
    for (int j = 0; j < kEssLags; ++j) part_lag[slice * block + li * kEssLags + j] = acc[j];
    __syncthreads();
    // base is odd: thread p has the pair of lags base + 2p, base + 2p + 1
    if (2 * threadIdx.x < static_cast<unsigned>(block)) {
      double a = 0.0, b = 0.0;
      for (int q = 0; q < slices; ++q) {
        const double2 v = *reinterpret_cast<const double2*>(part_lag + q * block + 2 * threadIdx.x);
        a += v.x;
        b += v.y;
      }
      const double pair = a / static_cast<double>(n) / var + b / static_cast<double>(n) / var;
      pairs[threadIdx.x] = pair;
      if ((base + 1) / 2 + threadIdx.x >= kmax || pair < 0.0) atomicMin(&first_negative, threadIdx.x);
    }
    __syncthreads();
    const int keep = first_negative;
    if (threadIdx.x == 0) {
      double tau = tau_sh;
      const int m = keep < block / 2 ? keep : block / 2;
#pragma unroll 8
      for (int p = 0; p < m; ++p) tau += 2.0 * pairs[p];
      tau_sh = tau;
    }
    if (keep < block / 2) break;
  }
  if (threadIdx.x == 0) {
    double tau = tau_sh < 1.0 ? 1.0 : tau_sh;
    ess[series] = static_cast<double>(n) / tau;
  }
}

// Split-R-hat of `group` coordinates per CTA.  A warp's lanes are coordinates
// by rows; `subs` half-chains at a time have 32 / subs warps each.  Their means
// stay in shared memory for the spread, or, where there are too many (keep
// false), are taken a second time: no scratch, whose allocation alone took
// 100 us after a synchronisation.  What bounds it is loads in flight, so
// each lane issues kRhatLoads before it adds: 700 x 16 series of 2,500 samples
// 160 -> 44 us (of 12,500: 419 -> 171), 50 x 4: 119 -> 15 us.
constexpr int kRhatThreads = 1024;
constexpr int kRhatWarps = kRhatThreads / 32;
constexpr int kRhatLoads = 8;
constexpr size_t kRhatMeans = 128 * 1024;  // bytes kept for the means
__global__ void __launch_bounds__(kRhatThreads) rhat_kernel(const float* __restrict__ s, long N, int dim, int nchains,
                                                            int layout, int lg_group, int subs, bool keep,
                                                            double* __restrict__ rhat) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ double part[kRhatWarps][8][2];
  __shared__ double round_mean[kRhatWarps][8], round_var[kRhatWarps][8];
  double* mean_sh = reinterpret_cast<double*>(sm);  // [half-chain][coordinate]
  const int group = 1 << lg_group, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane & (group - 1), warps = kRhatWarps / subs, sub = warp / warps;
  const int row0 = (warp % warps) * (32 >> lg_group) + (lane >> lg_group), rows = warps * (32 >> lg_group);
  const int dd = blockIdx.x * group + g;
  const long spc = N / nchains, half = spc / 2;
  const long step = static_cast<long>(layout == 0 ? 1 : nchains) * dim;
  const int m = 2 * nchains;
  // means and Bessel-corrected variances of half-chains j0 .. j0 + subs - 1
  auto round = [&](int j0) {
    double ps = 0.0, ps2 = 0.0;
    const int j = j0 + sub;
    if (dd < dim && j < m) {
      const float* src = s + series_row(layout, j / 2, (j % 2) * half, spc, nchains) * dim + dd;
      const long at = rows * step;
      const float* q = src + row0 * step;
      int i = row0;
      for (; i + (kRhatLoads - 1) * rows < half; i += kRhatLoads * rows, q += kRhatLoads * at) {
        float v[kRhatLoads];
#pragma unroll
        for (int u = 0; u < kRhatLoads; ++u) v[u] = q[u * at];
#pragma unroll
        for (int u = 0; u < kRhatLoads; ++u) {
          const double x = static_cast<double>(v[u]);
          ps += x;
          ps2 += x * x;
        }
      }
      for (; i < half; i += rows, q += at) {
        const double x = static_cast<double>(*q);
        ps += x;
        ps2 += x * x;
      }
    }
    for (int o = 16; o >= group; o >>= 1) {
      ps += __shfl_xor_sync(0xffffffffu, ps, o);
      ps2 += __shfl_xor_sync(0xffffffffu, ps2, o);
    }
    if (lane < group) {
      part[warp][lane][0] = ps;
      part[warp][lane][1] = ps2;
    }
    __syncthreads();
    if (threadIdx.x < subs * group) {
      const int q = threadIdx.x >> lg_group;
      double S = 0.0, S2 = 0.0;
      for (int w = q * warps; w < (q + 1) * warps; ++w) {
        S += part[w][g][0];
        S2 += part[w][g][1];
      }
      const double mean = S / half;
      const double var = (S2 / half) - mean * mean;
      round_mean[q][g] = mean;
      round_var[q][g] = var * half / (half - 1);
      if (keep && j0 + q < m) mean_sh[(j0 + q) * group + g] = mean;
    }
    __syncthreads();
  };
  double grand = 0.0, W = 0.0;  // thread g < group
  for (int j0 = 0; j0 < m; j0 += subs) {
    round(j0);
    if (threadIdx.x < group) {
      for (int q = 0; q < subs && j0 + q < m; ++q) {
        grand += round_mean[q][g];
        W += round_var[q][g];
      }
    }
  }
  // B: squared deviations from the grand mean
  const double gm = grand / m;
  double B = 0.0;
  for (int j0 = 0; j0 < m; j0 += subs) {
    if (!keep) round(j0);
    if (threadIdx.x < group) {
      for (int q = 0; q < subs && j0 + q < m; ++q) {
        const double mean = keep ? mean_sh[(j0 + q) * group + g] : round_mean[q][g];
        B += (mean - gm) * (mean - gm);
      }
    }
  }
  if (threadIdx.x < group && dd < dim) {
    B *= static_cast<double>(half) / (m - 1);
    W /= m;
    const double var_hat = ((half - 1.0) / half) * W + B / half;
    rhat[dd] = (W > 1e-30) ? sqrt(var_hat / W) : 1.0;
  }
}

}  // namespace
}  // namespace naja

using namespace naja;

extern "C" int naja_validate(const float* samples, long long N, int dim, int nchains, int layout, double* ess,
                             double* rhat, void* stream_ptr) {
  if (!samples || dim <= 0 || nchains <= 0 || N <= 0)
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_validate: bad arguments");
  if (layout != 0 && layout != 1) return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_validate: layout must be 0 or 1");
  if (N % nchains != 0)
    return fail(NAJA_ERR_RUNTIME, "n_total (" + std::to_string(N) + ") not divisible by n_chains (" +
                                      std::to_string(nchains) + ")");
  const long spc = static_cast<long>(N / nchains);
  if (ess && spc < 4) return fail(NAJA_ERR_INVALID_ARGUMENT, "compute_ess: fewer than 4 samples per chain");
  if (rhat && spc / 2 < 2) return fail(NAJA_ERR_INVALID_ARGUMENT, "compute_split_rhat: chain too short to split");
  if (ess && spc > kEssMaxSeries)
    return fail(NAJA_ERR_UNSUPPORTED, "naja_validate: more than " + std::to_string(kEssMaxSeries) +
                                          " samples per chain");
  if (int st = require_local("naja_validate", {samples, ess, rhat})) return st;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  DeviceBuffer bs, be, br;
  const void* ds = nullptr;
  int st = device_view(samples, static_cast<size_t>(N) * dim * sizeof(float), stream, bs, &ds);
  if (st) return st;
  double* de = ess;
  double* dr = rhat;
  const bool host_e = ess && !is_device_ptr(ess), host_r = rhat && !is_device_ptr(rhat);
  if (host_e) {
    if ((st = be.alloc(static_cast<size_t>(dim) * nchains * sizeof(double), stream))) return st;
    de = static_cast<double*>(be.ptr);
  }
  if (host_r) {
    if ((st = br.alloc(static_cast<size_t>(dim) * sizeof(double), stream))) return st;
    dr = static_cast<double*>(br.ptr);
  }
  if (ess) {
    const size_t smem = (static_cast<size_t>(spc) + kEssPad) * sizeof(float);
    // (one limit whatever the series: threads with different ones do not undo each other's)
    cudaFuncSetAttribute(ess_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>((kEssMaxSeries + kEssPad) * sizeof(float)));
    ess_kernel<<<dim * nchains, kEssThreads, smem, stream>>>(static_cast<const float*>(ds), static_cast<long>(N), dim,
                                                             nchains, layout, de);
  }
  if (rhat) {
    // eight coordinates per CTA (whole sectors of the rows), fewer where there
    // are no more; as many half-chains side by side as there are, up to a warp each
    int lg = 3, subs = 1;
    while (lg > 0 && (1 << (lg - 1)) >= dim) --lg;
    while (subs < kRhatWarps && subs < 2 * nchains) subs *= 2;
    const size_t means = (static_cast<size_t>(2) * nchains * sizeof(double)) << lg;
    const bool keep = means <= kRhatMeans;
    const size_t smem = keep ? means : 0;
    cudaFuncSetAttribute(rhat_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kRhatMeans));
    rhat_kernel<<<static_cast<unsigned>((dim + (1 << lg) - 1) >> lg), kRhatThreads, smem, stream>>>(
        static_cast<const float*>(ds), static_cast<long>(N), dim, nchains, layout, lg, subs, keep, dr);
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && host_e)
    e = cudaMemcpyAsync(ess, de, static_cast<size_t>(dim) * nchains * sizeof(double), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess && host_r)
    e = cudaMemcpyAsync(rhat, dr, static_cast<size_t>(dim) * sizeof(double), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess && (host_e || host_r || bs.ptr)) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("naja_validate: ") + cudaGetErrorString(e));
  return NAJA_OK;
}
