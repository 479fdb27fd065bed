// Kernels of the learned-rounding network (see include/naja_mlp.h).
//
// GEMM: D (M x N) = A (M x K) B (N x K)^T with BF16 operands and an FP32
// accumulator in tensor memory, persistent over 128 x TN output tiles
// (n fastest), one CTA per SM.  TN is 16, 32, 64 or 128: a training step's
// products are small (a batch of 64 rows against 512 or 23,100 outputs), so
// what bounds them is how many SMs take part and how many bytes each has in
// flight, and the widest tile that still gives every SM work is taken
// (gemm_tile_n).  The order of K is the same for every width, and so are the
// results.
//   warp 4, one thread : TMA producer, 2-D tiled loads (128-byte swizzle) of
//                        a 64-value K slice of A (128 rows, 64 where M <= 64)
//                        and of B per stage into a ring of up to 16 stages;
//                        loads past the matrix edges read zeros, so M, N and K
//                        need no padding.
//   warp 5, one thread : MMA issuer, 4 tcgen05.mma (K = 16 each) per stage
//                        into one of two accumulators (tiles alternate); the
//                        stage is released with tcgen05.commit.
//   warps 0-3          : epilogue, tcgen05.ld of their 32 accumulator lanes
//                        (one output row per thread), bias, GELU; row-major
//                        outputs go through a 32 x 33 block of shared memory
//                        so that a store covers 32 columns of a row, the
//                        transposed one is written as the lanes hold it.
// One training step (2600-512-512-23100, batch 64): the nine products took
// 480 us with 128 x 128 tiles and a row per thread in the stores, 188 us now.
// Every wait is bounded by the global timer; on expiry the CTA records an
// error in a device word (read by naja_mlp_check), stops issuing, drains its
// own copies and MMAs and frees its tensor memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>

#include "../../include/naja_chr.h"
#include "../../include/naja_mlp.h"
#include "capi_internal.cuh"
#include "common.cuh"
#include "tc_common.cuh"

namespace naja {
namespace {

constexpr int kTileM = 128;
constexpr int kMaxStages = 16;
constexpr int kStageSlices = 2;  // K slices per stage: one barrier round trip for both
constexpr int kThreads = 192;
constexpr uint64_t kTimeoutNs = 5ull * 1000 * 1000 * 1000;
constexpr int kStagePad = 32 * 33;  // floats of an epilogue warp's block
constexpr size_t kRingBudget = 200 * 1024;

enum GemmError : int { kGemmTimeoutLoad = 21, kGemmTimeoutSlot = 22, kGemmTimeoutAcc = 23, kGemmTimeoutEpi = 24 };

__device__ int g_gemm_err[4];

struct GemmArgs {
  int M, N, kslices, tiles_n;
  int stages, a_bytes;  // ring depth; bytes of A's slice (64 or 128 rows)
  long long tiles;
  naja_gemm_epilogue epi;
};

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * expf(-0.5f * x * x) * 0.39894228040143268f;
}

template <int TN>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
                     const __grid_constant__ GemmArgs a) {
  constexpr uint32_t kTmemCols = 2 * TN < 32 ? 32 : 2 * TN;
  constexpr uint32_t kBTile = TN * 128;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t slice_bytes = static_cast<uint32_t>(a.a_bytes) + kBTile;
  const uint32_t stage_bytes = kStageSlices * slice_bytes;
  const int S = a.stages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(S) * stage_bytes);
  uint64_t* empty = full + kMaxStages;
  uint64_t* acc_full = empty + kMaxStages;  // [2]
  uint64_t* acc_empty = acc_full + 2;       // [2]
  uint64_t* drain_bar = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* blocks = reinterpret_cast<float*>(smem + static_cast<size_t>(S) * stage_bytes + 512);
  int* err = g_gemm_err;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(&acc_full[q], 1);
      mbar_init(&acc_empty[q], 4);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tmem_slot, kTmemCols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;
  const int K = a.kslices;

  if (warp == 4) {
    if (lane == 0) {
      int stage = 0;
      uint32_t round = 0, last_parity = 0, used = 0;
      for (long long tile = blockIdx.x; tile < a.tiles && !*abort_flag; tile += gridDim.x) {
        const int tm = static_cast<int>(tile / a.tiles_n), tn = static_cast<int>(tile % a.tiles_n);
        for (int ks = 0; ks < K; ks += kStageSlices) {
          if (round >= 1 && !mbar_wait_bounded(&empty[stage], (round - 1) & 1u, kTimeoutNs)) {
            set_error(err, kGemmTimeoutSlot, static_cast<int>(blockIdx.x), stage, ks);
            *abort_flag = 1;
            break;
          }
          unsigned char* st = smem + static_cast<size_t>(stage) * stage_bytes;
          const int ns = min(kStageSlices, K - ks);
          mbar_arrive_expect_tx(&full[stage], ns * slice_bytes);
          for (int q = 0; q < ns; ++q) {
            tc::tma_load_2d(st + q * slice_bytes, &mA, (ks + q) * 64, tm * kTileM, &full[stage]);
            tc::tma_load_2d(st + q * slice_bytes + a.a_bytes, &mB, (ks + q) * 64, tn * TN, &full[stage]);
          }
          used |= 1u << stage;
          last_parity = (last_parity & ~(1u << stage)) | ((round & 1u) << stage);
          if (++stage == S) {
            stage = 0;
            ++round;
          }
        }
      }
      for (int s = 0; s < S; ++s)
        if (((used >> s) & 1u) && !mbar_wait_bounded(&full[s], (last_parity >> s) & 1u, kTimeoutNs))
          set_error(err, kGemmTimeoutLoad, static_cast<int>(blockIdx.x), s, -1);
    }
  } else if (warp == 5) {
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(kTileM, TN);
      int stage = 0;
      uint32_t parity = 0, acc_round = 0;
      bool issued = false;
      for (long long tile = blockIdx.x; tile < a.tiles && !*abort_flag; tile += gridDim.x) {
        const uint32_t buf = acc_round & 1u, use = acc_round >> 1;
        if (use >= 1 && !mbar_wait_bounded(&acc_empty[buf], (use - 1) & 1u, kTimeoutNs)) {
          set_error(err, kGemmTimeoutEpi, static_cast<int>(blockIdx.x), static_cast<int>(acc_round), -1);
          *abort_flag = 1;
          break;
        }
        tc::fence_after();
        bool ok = true;
        for (int ks = 0; ks < K; ks += kStageSlices) {
          if (!mbar_wait_bounded(&full[stage], parity, kTimeoutNs)) {
            set_error(err, kGemmTimeoutLoad, static_cast<int>(blockIdx.x), stage, ks);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc::fence_after();
          const unsigned char* st = smem + static_cast<size_t>(stage) * stage_bytes;
          // (with 64 rows of A, accumulator rows 64-127 come from whatever
          // follows them in shared memory and are not read)
          for (int q = 0; q < kStageSlices && ks + q < K; ++q, st += slice_bytes) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              tc::mma_bf16(tmem + buf * TN, tc::desc_sw128(st + kk * 32), tc::desc_sw128(st + a.a_bytes + kk * 32), idesc,
                           (ks + q > 0 || kk > 0) ? 1u : 0u);
            }
          }
          issued = true;
          tc::commit(&empty[stage]);
          if (++stage == S) {
            stage = 0;
            parity ^= 1u;
          }
        }
        if (!ok) break;
        tc::commit(&acc_full[buf]);
        ++acc_round;
      }
      if (issued) {
        tc::commit(drain_bar);
        if (!mbar_wait_bounded(drain_bar, 0u, kTimeoutNs))
          set_error(err, kGemmTimeoutAcc, static_cast<int>(blockIdx.x), -1, -1);
      }
    }
  } else {
    const naja_gemm_epilogue& e = a.epi;
    constexpr int CB = TN < 32 ? TN : 32;  // columns of an epilogue block
    float* blk = blocks + warp * kStagePad;
    uint32_t acc_round = 0;
    for (long long tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
      const uint32_t buf = acc_round & 1u, use = acc_round >> 1;
      const bool ok = mbar_wait_bounded(&acc_full[buf], use & 1u, kTimeoutNs);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) set_error(err, kGemmTimeoutAcc, static_cast<int>(blockIdx.x), warp, static_cast<int>(acc_round));
        *abort_flag = 1;
        break;
      }
      tc::fence_after();
      const int tm = static_cast<int>(tile / a.tiles_n), tn = static_cast<int>(tile % a.tiles_n);
      const int row0 = tm * kTileM + warp * 32;
      const int rows = min(32, a.M - row0);  // of this warp; may be <= 0
      if (rows > 0) {
#pragma unroll 1
        for (int c = 0; c < TN; c += CB) {
          uint32_t r[CB];
          const uint32_t at = tmem + (static_cast<uint32_t>(warp * 32) << 16) + buf * TN + static_cast<uint32_t>(c);
          if constexpr (CB == 32) tc::tmem_ld32(at, r);
          else tc::tmem_ld16(at, r);
          const int n0 = tn * TN + c;
          const int cols = min(CB, a.N - n0);
          if (cols <= 0) break;
          if (e.bias) {
#pragma unroll
            for (int q = 0; q < CB; ++q)
              if (q < cols) r[q] = __float_as_uint(__uint_as_float(r[q]) + e.bias[n0 + q]);
          }
          // 32 columns (or the 16 of a narrow tile twice: two rows per pass)
          // of a row per store
          constexpr int RP = 32 / CB;
          const int lc = lane % CB, lr = lane / CB;
          if (e.c_f32) {
#pragma unroll
            for (int q = 0; q < CB; ++q) blk[lane * 33 + q] = __uint_as_float(r[q]);
            __syncwarp();
            if (lc < cols) {
#pragma unroll 8
              for (int j = lr; j < rows; j += RP) {
                float* cp = e.c_f32 + static_cast<size_t>(row0 + j) * e.ldc + n0 + lc;
                const float v = blk[j * 33 + lc];
                *cp = e.accumulate ? *cp + v : v;
              }
            }
            __syncwarp();
          }
          if (e.act || e.act_t) {
            if (e.gelu) {
#pragma unroll
              for (int q = 0; q < CB; ++q) r[q] = __float_as_uint(gelu_f(__uint_as_float(r[q])));
            }
            if (e.act_t && lane < rows) {
#pragma unroll
              for (int q = 0; q < CB; ++q)
                if (q < cols)
                  reinterpret_cast<__nv_bfloat16*>(e.act_t)[static_cast<size_t>(n0 + q) * e.ld_act_t + row0 + lane] =
                      __float2bfloat16_rn(__uint_as_float(r[q]));
            }
            if (e.act) {
#pragma unroll
              for (int q = 0; q < CB; ++q) blk[lane * 33 + q] = __uint_as_float(r[q]);
              __syncwarp();
              if (lc < cols) {
#pragma unroll 8
                for (int j = lr; j < rows; j += RP)
                  reinterpret_cast<__nv_bfloat16*>(e.act)[static_cast<size_t>(row0 + j) * e.ld_act + n0 + lc] =
                      __float2bfloat16_rn(blk[j * 33 + lc]);
              }
              __syncwarp();
            }
          }
        }
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
      ++acc_round;
    }
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == 0) tc::tmem_dealloc(tmem, kTmemCols);
}

// The tile width that takes the fewest cycles by this account, the narrowest
// of equals: a CTA's tiles follow one another, each as long as the longer of
// its slices' way into shared memory (61 bytes a cycle) and its epilogue (28
// cycles a column), which overlap, and 380 cycles to start; the shorter of the
// two stands alone once.  us at 16 / 32 / 64 / 128 columns: 4096 x 512 x 23100
// 620 / 364 / 192 / 113, 2048 x 512 x 2600 53 / 32 / 24 / 30, 64 x 512 x 23100
// 98 / 98 / 100 / 102, 512 x 2600 x 64 17.0 / 15.8 / 16.9 / 16.3; the widest
// tile that makes two per SM, whatever K, took 364 and 53 us for the first two.
int gemm_tile_n(int M, int N, int K, int a_rows, int sms) {
  const long long rows = (M + kTileM - 1) / kTileM, slices = (K + 63) / 64;
  int best = 16;
  long long least = 0;
  for (int tn : {16, 32, 64, 128}) {
    const long long rounds = (rows * ((N + tn - 1) / tn) + sms - 1) / sms;
    const long long load = slices * (a_rows * 128 + tn * 128) / 61, store = 28 * tn;
    const long long cycles = rounds * (std::max(load, store) + 380) + std::min(load, store);
    if (least == 0 || cycles < least) {
      least = cycles;
      best = tn;
    }
  }
  return best;
}

template <int TN>
cudaError_t gemm_launch(const CUtensorMap& mA, const CUtensorMap& mB, GemmArgs a, int sms, cudaStream_t stream) {
  const size_t stage = kStageSlices * (static_cast<size_t>(a.a_bytes) + TN * 128);
  a.stages = static_cast<int>(std::min<size_t>(kMaxStages, kRingBudget / stage));
  a.tiles_n = (a.N + TN - 1) / TN;
  a.tiles = static_cast<long long>((a.M + kTileM - 1) / kTileM) * a.tiles_n;
  // the MMA reads 128 rows of A from the last stage on: the blocks behind the
  // ring are more than the 64 rows that may be missing there
  constexpr size_t beside = 1024 + 512 + 4 * kStagePad * sizeof(float);
  const size_t smem = a.stages * stage + beside;
  const cudaError_t e =
      // (one limit whatever the product: threads with different ones do not undo each other's)
      cudaFuncSetAttribute(gemm_bf16_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kRingBudget + beside));
  if (e != cudaSuccess) return e;
  const int grid = static_cast<int>(std::min<long long>(sms, a.tiles));
  gemm_bf16_kernel<TN><<<grid, kThreads, smem, stream>>>(mA, mB, a);
  return cudaSuccess;
}

// ------------------------------------------------------------ elementwise
// op(r, c) over a rows x cols matrix in 32 x 32 tiles; the FP32 value it
// returns is rounded to BF16 and written row-major (dst) and transposed
// (dst_t), either one optional, the latter through shared memory so that both
// stores cover whole rows.  What bounds these kernels is memory; transposing
// stores of two bytes each took twice the time of everything else in the Adam
// step of the 23,100 x 512 layer (143 us, 78 us now; 59 us at the
// measured copy rate).
constexpr int kTile = 32;
template <class Op>
__device__ __forceinline__ void for_tile(int rows, int cols, Op&& op, __nv_bfloat16* dst, int ld, __nv_bfloat16* dst_t,
                                         int ld_t) {
  __shared__ __nv_bfloat16 t[kTile][kTile + 2];
  const int tiles_c = (cols + kTile - 1) / kTile;
  const int r0 = blockIdx.x / tiles_c * kTile, c0 = blockIdx.x % tiles_c * kTile;
  const int x = threadIdx.x % kTile, y = threadIdx.x / kTile;  // 256 threads: 8 rows per pass
  const int c = c0 + x;
#pragma unroll 4
  for (int i = y; i < kTile; i += 8) {
    const int r = r0 + i;
    if (r < rows && c < cols) {
      const __nv_bfloat16 b = __float2bfloat16_rn(op(r, c));
      if (dst) dst[static_cast<size_t>(r) * ld + c] = b;
      t[i][x] = b;
    }
  }
  if (dst_t) {
    __syncthreads();
    const int r = r0 + x;
#pragma unroll 4
    for (int i = y; i < kTile; i += 8)
      if (r < rows && c0 + i < cols) dst_t[static_cast<size_t>(c0 + i) * ld_t + r] = t[x][i];
  }
}

__global__ void __launch_bounds__(256) cast_bf16_kernel(int rows, int cols, const float* __restrict__ src, int ld_src,
                                                        __nv_bfloat16* dst, int ld_dst, __nv_bfloat16* dst_t,
                                                        int ld_dst_t) {
  for_tile(rows, cols, [&](int r, int c) { return src[static_cast<size_t>(r) * ld_src + c]; }, dst, ld_dst, dst_t,
           ld_dst_t);
}

__global__ void __launch_bounds__(256)
    gelu_backward_kernel(int rows, int cols, const float* __restrict__ dact, const float* __restrict__ pre, int ld,
                         float* dpre, __nv_bfloat16* dpre_bf, int ld_bf, __nv_bfloat16* dpre_bf_t, int ld_bf_t) {
  for_tile(
      rows, cols,
      [&](int r, int c) {
        const size_t o = static_cast<size_t>(r) * ld + c;
        const float g = dact[o] * gelu_grad_f(pre[o]);
        if (dpre) dpre[o] = g;
        return g;
      },
      dpre_bf, ld_bf, dpre_bf_t, ld_bf_t);
}

__global__ void __launch_bounds__(256)
    mse_grad_kernel(int rows, int cols, const float* __restrict__ out, const float* __restrict__ target, int ld,
                    const float* __restrict__ w, double* loss, float* grad, __nv_bfloat16* grad_bf, int ld_bf,
                    __nv_bfloat16* grad_bf_t, int ld_bf_t) {
  __shared__ double part[8];
  double acc = 0.0;
  const float inv_rows = 1.0f / static_cast<float>(rows);
  for_tile(
      rows, cols,
      [&](int r, int c) {
        const size_t o = static_cast<size_t>(r) * ld + c;
        const float wc = w ? w[c] : 1.0f;
        const float diff = out[o] - target[o];
        acc += static_cast<double>(wc) * diff * diff;
        const float g = 2.0f * wc * diff * inv_rows;
        if (grad) grad[o] = g;
        return g;
      },
      grad_bf, ld_bf, grad_bf_t, ld_bf_t);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < 8; ++k) s += part[k];
    atomicAdd(loss, s / rows);
  }
}

__global__ void col_sum_kernel(int rows, int cols, const float* __restrict__ d, int ld, float* db) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  float s = 0.0f;
  // (in row order; the loads of 16 rows are in flight together)
#pragma unroll 16
  for (int r = 0; r < rows; ++r) s += d[static_cast<size_t>(r) * ld + c];
  db[c] = s;
}

__global__ void __launch_bounds__(256)
    adam_kernel(int rows, int cols, float* W, const float* __restrict__ g, float* m, float* v, int ld, float lr, float b1,
                float b2, float eps, float c1, float c2, __nv_bfloat16* w_bf, int ld_bf, __nv_bfloat16* w_bf_t,
                int ld_bf_t) {
  for_tile(
      rows, cols,
      [&](int r, int c) {
        const size_t o = static_cast<size_t>(r) * ld + c;
        const float gi = g[o];
        const float mi = b1 * m[o] + (1.0f - b1) * gi;
        const float vi = b2 * v[o] + (1.0f - b2) * gi * gi;
        m[o] = mi;
        v[o] = vi;
        const float wi = W[o] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
        W[o] = wi;
        return wi;
      },
      w_bf, ld_bf, w_bf_t, ld_bf_t);
}

// Blocks of a for_tile kernel.
unsigned tiles_for(int rows, int cols) {
  return static_cast<unsigned>((rows + kTile - 1) / kTile) * static_cast<unsigned>((cols + kTile - 1) / kTile);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int launch_status(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return NAJA_OK;
}

}  // namespace
}  // namespace naja

using namespace naja;

extern "C" {

int naja_gemm_bf16(int M, int N, int K, const void* A, int lda, const void* B, int ldb,
                   const naja_gemm_epilogue* epi, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !epi) return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_gemm_bf16: bad arguments");
  if (lda < K || ldb < K || (lda % 8) || (ldb % 8) || !aligned16(A) || !aligned16(B))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_gemm_bf16: BF16 rows must be 16-byte aligned with pitch >= K");
  if ((epi->c_f32 && epi->ldc < N) || (epi->act && epi->ld_act < N) || (epi->act_t && epi->ld_act_t < M))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_gemm_bf16: epilogue pitch too small");
  if (int st = require_local("naja_gemm_bf16", {A, B, epi->bias, epi->c_f32, epi->act, epi->act_t})) return st;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int a_rows = M <= 64 ? 64 : kTileM, tn = gemm_tile_n(M, N, K, a_rows, sms);
  CUtensorMap mA, mB;
  if (!tc::make_map_bf16(&mA, A, M, K, lda, a_rows) || !tc::make_map_bf16(&mB, B, N, K, ldb, tn))
    return fail(NAJA_ERR_CUDA, "naja_gemm_bf16: cuTensorMapEncodeTiled failed");
  GemmArgs a;
  a.M = M;
  a.N = N;
  a.kslices = (K + 63) / 64;
  a.a_bytes = a_rows * 128;
  a.epi = *epi;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = tn == 128  ? gemm_launch<128>(mA, mB, a, sms, s)
                        : tn == 64 ? gemm_launch<64>(mA, mB, a, sms, s)
                        : tn == 32 ? gemm_launch<32>(mA, mB, a, sms, s)
                                   : gemm_launch<16>(mA, mB, a, sms, s);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("naja_gemm_bf16: ") + cudaGetErrorString(e));
  return launch_status("naja_gemm_bf16");
}

int naja_mlp_check(void* stream) {
  int w[4] = {0, 0, 0, 0};
  cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(w, g_gemm_err, sizeof(w));
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("naja_mlp_check: ") + cudaGetErrorString(e));
  if (w[0] != 0) {
    const int z[4] = {0, 0, 0, 0};
    cudaMemcpyToSymbol(g_gemm_err, z, sizeof(z));
    return fail(NAJA_ERR_DEVICE, "naja_gemm_bf16: tensor-core pipeline gave up a bounded wait (code " +
                                     std::to_string(w[0]) + ", " + std::to_string(w[1]) + ", " + std::to_string(w[2]) +
                                     ", " + std::to_string(w[3]) + ")");
  }
  return NAJA_OK;
}

int naja_cast_bf16(int rows, int cols, const float* src, int ld_src, void* dst, int ld_dst, void* dst_t,
                   int ld_dst_t, void* stream) {
  if (rows <= 0 || cols <= 0 || !src || ld_src < cols || (dst && ld_dst < cols) || (dst_t && ld_dst_t < rows))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_cast_bf16: bad arguments");
  if (int st = require_local("naja_cast_bf16", {src, dst, dst_t})) return st;
  cast_bf16_kernel<<<tiles_for(rows, cols), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      rows, cols, src, ld_src, static_cast<__nv_bfloat16*>(dst), ld_dst, static_cast<__nv_bfloat16*>(dst_t), ld_dst_t);
  return launch_status("naja_cast_bf16");
}

int naja_gelu_backward(int rows, int cols, const float* dact, const float* pre, int ld, float* dpre, void* dpre_bf,
                       int ld_bf, void* dpre_bf_t, int ld_bf_t, void* stream) {
  if (rows <= 0 || cols <= 0 || !dact || !pre || ld < cols || (dpre_bf && ld_bf < cols) || (dpre_bf_t && ld_bf_t < rows))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_gelu_backward: bad arguments");
  if (int st = require_local("naja_gelu_backward", {dact, pre, dpre, dpre_bf, dpre_bf_t})) return st;
  gelu_backward_kernel<<<tiles_for(rows, cols), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      rows, cols, dact, pre, ld, dpre, static_cast<__nv_bfloat16*>(dpre_bf), ld_bf,
      static_cast<__nv_bfloat16*>(dpre_bf_t), ld_bf_t);
  return launch_status("naja_gelu_backward");
}

int naja_mse_grad(int rows, int cols, const float* out, const float* target, int ld, const float* w, double* loss,
                  float* grad, void* grad_bf, int ld_bf, void* grad_bf_t, int ld_bf_t, void* stream) {
  if (rows <= 0 || cols <= 0 || !out || !target || !loss || ld < cols || (grad_bf && ld_bf < cols) ||
      (grad_bf_t && ld_bf_t < rows))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_mse_grad: bad arguments");
  if (int st = require_local("naja_mse_grad", {out, target, w, loss, grad, grad_bf, grad_bf_t})) return st;
  mse_grad_kernel<<<tiles_for(rows, cols), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      rows, cols, out, target, ld, w, loss, grad, static_cast<__nv_bfloat16*>(grad_bf), ld_bf,
      static_cast<__nv_bfloat16*>(grad_bf_t), ld_bf_t);
  return launch_status("naja_mse_grad");
}

int naja_col_sum(int rows, int cols, const float* d, int ld, float* db, void* stream) {
  if (rows <= 0 || cols <= 0 || !d || !db || ld < cols) return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_col_sum: bad arguments");
  if (int st = require_local("naja_col_sum", {d, db})) return st;
  col_sum_kernel<<<(cols + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(rows, cols, d, ld, db);
  return launch_status("naja_col_sum");
}

int naja_adam(int rows, int cols, float* W, const float* g, float* m, float* v, int ld, float lr, float beta1,
              float beta2, float eps, int step, void* w_bf, int ld_bf, void* w_bf_t, int ld_bf_t, void* stream) {
  if (rows <= 0 || cols <= 0 || !W || !g || !m || !v || ld < cols || step < 1 || (w_bf && ld_bf < cols) ||
      (w_bf_t && ld_bf_t < rows))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_adam: bad arguments");
  if (int st = require_local("naja_adam", {W, g, m, v, w_bf, w_bf_t})) return st;
  const float c1 = 1.0f / (1.0f - std::pow(beta1, static_cast<float>(step)));
  const float c2 = 1.0f / (1.0f - std::pow(beta2, static_cast<float>(step)));
  adam_kernel<<<tiles_for(rows, cols), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      rows, cols, W, g, m, v, ld, lr, beta1, beta2, eps, c1, c2, static_cast<__nv_bfloat16*>(w_bf), ld_bf,
      static_cast<__nv_bfloat16*>(w_bf_t), ld_bf_t);
  return launch_status("naja_adam");
}

}  // extern "C"
