// Device-side `naja validate` metrics: Geyer ESS per (dim, chain) and
// split-R-hat per dim, following src/validate/mcmc.cpp:17-194 of
// quothbonney/naja.
//
// ESS: one CTA per chain and group of coordinates (whole 32-byte sectors of
// the sample rows).  Each series is centred in shared memory and its
// autocovariances are summed directly (FP32 products, FP64 sums) in blocks of
// 64 lags until Geyer's initial positive sequence stops.  The reference
// obtains the same acov[k] = (1/n) sum (x_t-m)(x_{t+k}-m) from a float FFT of
// size 2n; the direct sum needs only the lags the rule reaches (a few blocks
// for a mixing chain) and has no FFT round-off.
//
// R-hat: half-chain sums in FP64 as mcmc.cpp takes them, over sample rows as
// they lie in memory (a lane per coordinate), then one combination.
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

// Lags of a block, lags per thread (a sliding window: one new value per
// sample for kEssLags products) and the slices of a series that the threads of
// one lag group share out.
constexpr int kEssBlock = 64;
constexpr int kEssLags = 4;
constexpr int kEssLanes = kEssBlock / kEssLags;
constexpr int kEssSlices = kEssThreads / kEssLanes;
constexpr int kEssPad = kEssBlock + 4;  // zeros behind a series: a product past its end is 0

// Floats between the series of a CTA: four values of eight series fall on
// distinct banks.
__host__ __device__ inline long ess_pitch(long n) { return (n + kEssPad + 27) / 32 * 32 + 4; }

// What bounds it is the conversion of each FP32 product to FP64 (16 per clock
// and SM), so the gain is in the products not taken: blocks of 64 lags instead
// of 512 (16 chains x 2,500 samples x 700 coordinates, correlations 0.3 to
// 0.99, ESS and R-hat with their copies: 3.56 -> 1.71 ms).
__global__ void __launch_bounds__(kEssThreads) ess_kernel(const float* __restrict__ s, long N, int dim, int nchains,
                                                        int layout, int group, double* __restrict__ ess) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ double scratch[32];
  __shared__ double part_lag[kEssSlices][kEssBlock];
  __shared__ double acov[kEssBlock];
  __shared__ int stop_flag;
  __shared__ double tau_sh;
  float* all = reinterpret_cast<float*>(sm);
  const long n = N / nchains, pitch = ess_pitch(n);
  const int c = blockIdx.x % nchains, dd0 = blockIdx.x / nchains * group;
  const int ng = dim - dd0 < group ? dim - dd0 : group;
  for (long e = threadIdx.x; e < n * group; e += kEssThreads) {
    const long i = e / group;
    const int g = static_cast<int>(e - i * group);
    if (g < ng) all[g * pitch + i] = s[series_row(layout, c, i, n, nchains) * dim + dd0 + g];
  }
  for (int e = threadIdx.x; e < group * kEssPad; e += kEssThreads)
    all[(e / kEssPad) * pitch + n + e % kEssPad] = 0.0f;
  __syncthreads();
  const int li = threadIdx.x % kEssLanes, slice = threadIdx.x / kEssLanes;
  for (int g = 0; g < ng; ++g) {
    float* y = all + g * pitch;
    const long series = static_cast<long>(dd0 + g) * nchains + c;
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
      continue;
    }
    if (threadIdx.x == 0) {
      stop_flag = 0;
      tau_sh = 1.0;
    }
    __syncthreads();
    // pair k uses lags 2k-1, 2k, for k = 1 .. kmax-1
    const long kmax = n / 2;
    for (long base = 1; base <= 2 * (kmax - 1); base += kEssBlock) {
      // this thread: lags lag0 .. lag0 + 3 over its slice of t < n - base
      // (beyond that every product is 0)
      const long lag0 = base + li * kEssLags, len = n - base;
      const long t0 = len * slice / kEssSlices, t1 = len * (slice + 1) / kEssSlices;
      double acc[kEssLags];
#pragma unroll
      for (int j = 0; j < kEssLags; ++j) acc[j] = 0.0;
      // (a window past the padding only holds lags past n - 1: not summed)
      if (t0 < t1 && lag0 < n) {
        const long tend = t1 < n + kEssPad - lag0 - kEssLags ? t1 : n + kEssPad - lag0 - kEssLags;
        const float* yk = y + lag0;
        float w[kEssLags];
#pragma unroll
        for (int j = 0; j < kEssLags; ++j) w[j] = yk[t0 + j];
        long t = t0;
        for (; t + kEssLags <= tend; t += kEssLags) {
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
        for (; t < tend; ++t) {
          const float v = y[t];
#pragma unroll
          for (int j = 0; j < kEssLags; ++j) acc[j] += static_cast<double>(v * yk[t + j]);
        }
      }
#pragma unroll
      for (int j = 0; j < kEssLags; ++j) part_lag[slice][li * kEssLags + j] = acc[j];
      __syncthreads();
      if (threadIdx.x < kEssBlock) {
        double a = 0.0;
#pragma unroll
        for (int q = 0; q < kEssSlices; ++q) a += part_lag[q][threadIdx.x];
        acov[threadIdx.x] = a / static_cast<double>(n);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        double tau = tau_sh;
        // acov[i] holds lag base + i; base is odd, so pairs are (i, i+1) for even i.
        for (int i = 0; i < kEssBlock; i += 2) {
          const long k = (base + i + 1) / 2;
          if (k >= kmax) {
            stop_flag = 1;
            break;
          }
          const double pair = acov[i] / var + acov[i + 1] / var;
          if (pair < 0.0) {
            stop_flag = 1;
            break;
          }
          tau += 2.0 * pair;
        }
        tau_sh = tau;
      }
      __syncthreads();
      if (stop_flag) break;
    }
    if (threadIdx.x == 0) {
      double tau = tau_sh < 1.0 ? 1.0 : tau_sh;
      ess[series] = static_cast<double>(n) / tau;
    }
    __syncthreads();
  }
}

// Sums and sums of squares of half-chain j (blockIdx.x % 2k) for 32 coordinates,
// sums[(j * dim + dd) * 2].
__global__ void __launch_bounds__(256) rhat_sums_kernel(const float* __restrict__ s, long N, int dim, int nchains,
                                                        int layout, double* __restrict__ sums) {
  __shared__ double part[2][8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x % (2 * nchains), dd = blockIdx.x / (2 * nchains) * 32 + lane, c = j / 2, h = j % 2;
  const long spc = N / nchains, half = spc / 2;
  double ps = 0.0, ps2 = 0.0;
  if (dd < dim) {
#pragma unroll 4
    for (long i = w; i < half; i += 8) {
      const double v = static_cast<double>(s[series_row(layout, c, h * half + i, spc, nchains) * dim + dd]);
      ps += v;
      ps2 += v * v;
    }
  }
  part[0][w][lane] = ps;
  part[1][w][lane] = ps2;
  __syncthreads();
  if (w < 2 && dd < dim) {
    double t = 0.0;
    for (int q = 0; q < 8; ++q) t += part[w][q][lane];
    sums[(static_cast<size_t>(j) * dim + dd) * 2 + w] = t;
  }
}

__global__ void rhat_kernel(const double* __restrict__ sums, long N, int dim, int nchains, double* __restrict__ rhat) {
  const int dd = blockIdx.x * blockDim.x + threadIdx.x;
  if (dd >= dim) return;
  const long half = N / nchains / 2;
  const int m = 2 * nchains;
  double grand = 0.0, W = 0.0;
  // half-chain means and Bessel-corrected variances
  for (int j = 0; j < m; ++j) {
    const double* q = sums + (static_cast<size_t>(j) * dim + dd) * 2;
    const double mean = q[0] / half;
    double var = (q[1] / half) - mean * mean;
    var = var * half / (half - 1);
    grand += mean;
    W += var;
  }
  // B: squared deviations from the grand mean
  const double gm = grand / m;
  double B = 0.0;
  for (int j = 0; j < m; ++j) {
    const double mean = sums[(static_cast<size_t>(j) * dim + dd) * 2] / half;
    B += (mean - gm) * (mean - gm);
  }
  B *= static_cast<double>(half) / (m - 1);
  W /= m;
  const double var_hat = ((half - 1.0) / half) * W + B / half;
  rhat[dd] = (W > 1e-30) ? sqrt(var_hat / W) : 1.0;
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
  DeviceBuffer bs, be, br, bsum;
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
  if (rhat && (st = bsum.alloc(static_cast<size_t>(4) * nchains * dim * sizeof(double), stream))) return st;
  if (ess) {
    // eight coordinates per CTA (whole sectors) where they leave room for
    // another CTA, fewer for long series
    int group = 8;
    while (group > 1 && group * ess_pitch(spc) * sizeof(float) > (group > 4 ? 100u : 200u) * 1024) group /= 2;
    const size_t smem = group * ess_pitch(spc) * sizeof(float);
    cudaFuncSetAttribute(ess_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    ess_kernel<<<static_cast<unsigned>((dim + group - 1) / group) * nchains, kEssThreads, smem, stream>>>(
        static_cast<const float*>(ds), static_cast<long>(N), dim, nchains, layout, group, de);
  }
  if (rhat) {
    rhat_sums_kernel<<<static_cast<unsigned>((dim + 31) / 32) * 2 * nchains, 256, 0, stream>>>(
        static_cast<const float*>(ds), static_cast<long>(N), dim, nchains, layout, static_cast<double*>(bsum.ptr));
    rhat_kernel<<<(dim + 127) / 128, 128, 0, stream>>>(static_cast<const double*>(bsum.ptr), static_cast<long>(N), dim,
                                                       nchains, dr);
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
