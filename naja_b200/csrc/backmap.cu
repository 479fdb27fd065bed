// Backmap V = T Y + shift (reduced -> original flux space), the reference's
// backmap_into (src/gpu/backmap.cu:20-48 of quothbonney/naja: cublasDgemm
// followed by add_shift_cols_kernel) as one kernel with the shift fused into
// the epilogue.
//
// Layouts: T is n x d column-major (leading dimension ldt).  Y holds N
// samples as rows of d values (the sampler's output, row = sample), V
// receives N rows of n values -- the `samples.npy` layout of the
// back-transformed file.  In GEMM terms V (N x n) = Y (N x d) T^T (d x n).
//
// Modes (NAJA_BACKMAP_*):
//   FP64    FP64 tensor-core tiles (the reference's arithmetic, different
//           summation order than cuBLAS).
//   BF16X3  / TF32X3: split-precision tensor-core products on tcgen05,
//           in backmap_tc.cu.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/naja_chr.h"
#include "capi_internal.cuh"

namespace naja {

namespace {

// The FP64 product on the FP64 tensor cores (mma.sync m16n8k8): a CTA takes a
// 128 x 64 tile of V, eight warps of 32 x 32 each, and streams 16-deep slices
// of Y and T through a ring of kStages in shared memory (cp.async), Y in its
// own type and converted as the fragments are read.  What bounds it is the
// FP64 pipe: per slice a warp issues 16 products of 1,024 multiply-adds and 48
// shared-memory reads, whose pitches are free of bank conflicts.  The 4 x 4
// per thread kernel with scalar shared-memory reads it replaces was bound by
// those reads.  N 40,000, n = d = 700: 4.30 -> 1.32 ms (9.1 -> 29.8 TFLOP/s of
// about 37).
constexpr int kBM = 128;  // samples per CTA tile
constexpr int kBN = 64;   // outputs (rows of T) per CTA tile
constexpr int kBK = 16;
constexpr int kStages = 4;
constexpr int kYPitch = 20;                         // 8 rows x 4 columns on distinct banks
constexpr int kTPitch = 68;                         // 4 rows x 4 columns on distinct banks

template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src, bool ok) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(ok ? BYTES : 0)
                 : "memory");
}

// Copies a ROWS x COLS block whose rows are `ld` elements apart, from
// (row0, col0), rows below `rows` and columns below `cols` (zeros beyond).
// WIDE: 16-byte pieces (every row 16-byte aligned, cols and col0 multiples of
// a piece, so a piece is inside or outside as a whole).
template <class E, int ROWS, int COLS, int PITCH, bool WIDE>
__device__ __forceinline__ void load_block(E* dst, const E* src, long long ld, long long row0, long long rows, int col0,
                                           int cols) {
  constexpr int W = WIDE ? 16 / static_cast<int>(sizeof(E)) : 1, PER = COLS / W;
  for (int e = threadIdx.x; e < ROWS * PER; e += 256) {
    const int r = e / PER, c = e % PER * W;
    const bool ok = row0 + r < rows && col0 + c < cols;
    copy_async<W * static_cast<int>(sizeof(E))>(dst + r * PITCH + c, ok ? src + (row0 + r) * ld + col0 + c : src, ok);
  }
}

__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

template <class YT>
constexpr size_t fp64_smem_bytes() {
  return kStages * (kBM * kYPitch * sizeof(YT) + kBK * kTPitch * sizeof(double));
}

template <class YT, class VT, bool WIDE>
__global__ void __launch_bounds__(256, 2) backmap_fp64_kernel(int n, int d, long long N, const double* __restrict__ T,
                                                              int ldt, const double* __restrict__ shift,
                                                              const YT* __restrict__ Y, VT* __restrict__ V) {
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr int YP = kYPitch;
  YT* ys = reinterpret_cast<YT*>(sm);
  double* ts = reinterpret_cast<double*>(sm + kStages * kBM * YP * sizeof(YT));
  const long long s0 = static_cast<long long>(blockIdx.y) * kBM + static_cast<long long>(blockIdx.z) * 65535 * kBM;
  const int i0 = blockIdx.x * kBN;
  if (s0 >= N) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int wm = (warp & 3) * 32, wn = (warp >> 2) * 32;
  const int slices = (d + kBK - 1) / kBK;
  auto fetch = [&](int k) {
    if (k < slices) {
      const int st = k % kStages;
      load_block<YT, kBM, kBK, YP, WIDE>(ys + st * kBM * YP, Y, d, s0, N, k * kBK, d);
      load_block<double, kBK, kBN, kTPitch, WIDE>(ts + st * kBK * kTPitch, T, ldt, k * kBK, d, i0, n);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int k = 0; k < kStages - 1; ++k) fetch(k);
  double acc[2][4][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.0;
  for (int k = 0; k < slices; ++k) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // slice k has landed, and everyone is done with the one fetched over next
    fetch(k + kStages - 1);
    const YT* yt = ys + k % kStages * kBM * YP;
    const double* tt = ts + k % kStages * kBK * kTPitch;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 8) {
      double a[2][4], b[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int r = 0; r < 4; ++r)
          a[i][r] = static_cast<double>(yt[(wm + i * 16 + g + (r & 1) * 8) * YP + kk + q + (r >> 1) * 4]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int r = 0; r < 2; ++r) b[j][r] = tt[(kk + q + r * 4) * kTPitch + wn + j * 8 + g];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(acc[i][j], a[i], b[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long s = s0 + wm + i * 16 + g + h * 8;
      if (s >= N) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int o = i0 + wn + j * 8 + q * 2 + c;
          if (o < n) V[s * n + o] = static_cast<VT>(acc[i][j][2 * h + c] + shift[o]);
        }
    }
}

template <class YT, class VT, bool WIDE>
int launch_fp64_as(int n, int d, long long N, const double* T, int ldt, const double* shift, const void* Y, void* V,
                   cudaStream_t stream) {
  auto kern = backmap_fp64_kernel<YT, VT, WIDE>;
  constexpr int smem = static_cast<int>(fp64_smem_bytes<YT>());
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return NAJA_ERR_CUDA;
  // outputs fastest, so that a block of samples stays in L2 across its tiles
  const long long rows = (N + kBM - 1) / kBM;
  const dim3 grid(static_cast<unsigned>((n + kBN - 1) / kBN), static_cast<unsigned>(rows < 65535 ? rows : 65535),
                  static_cast<unsigned>((rows + 65534) / 65535));
  kern<<<grid, 256, smem, stream>>>(n, d, N, T, ldt, shift, static_cast<const YT*>(Y), static_cast<VT*>(V));
  return cudaGetLastError() == cudaSuccess ? NAJA_OK : NAJA_ERR_CUDA;
}

template <class YT, class VT>
int launch_fp64(int n, int d, long long N, const double* T, int ldt, const double* shift, const void* Y, void* V,
                cudaStream_t stream) {
  // 16-byte copies where every row of Y and T starts and ends on 16 bytes
  const auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  const bool wide = aligned(Y) && aligned(T) && d * sizeof(YT) % 16 == 0 && ldt % 2 == 0 && n % 2 == 0;
  return wide ? launch_fp64_as<YT, VT, true>(n, d, N, T, ldt, shift, Y, V, stream)
              : launch_fp64_as<YT, VT, false>(n, d, N, T, ldt, shift, Y, V, stream);
}

}  // namespace

int backmap_fp64_enqueue(int n, int d, long long N, const double* T, int ldt, const double* shift, const void* Y,
                         int y_dtype, void* V, int v_dtype, cudaStream_t stream) {
  int st;
  if (y_dtype == NAJA_DTYPE_F32)
    st = v_dtype == NAJA_DTYPE_F32 ? launch_fp64<float, float>(n, d, N, T, ldt, shift, Y, V, stream)
                                   : launch_fp64<float, double>(n, d, N, T, ldt, shift, Y, V, stream);
  else
    st = v_dtype == NAJA_DTYPE_F32 ? launch_fp64<double, float>(n, d, N, T, ldt, shift, Y, V, stream)
                                   : launch_fp64<double, double>(n, d, N, T, ldt, shift, Y, V, stream);
  if (st) return fail(st, std::string("backmap: launch failed: ") + cudaGetErrorString(cudaGetLastError()));
  return NAJA_OK;
}

}  // namespace naja

using namespace naja;

extern "C" int naja_backmap(int n, int d, long long N, const double* T, int ldt, const double* shift, const void* Y,
                            int y_dtype, void* V, int v_dtype, int mode, void* stream_ptr) {
  if (n <= 0 || d <= 0 || N < 0) return fail(NAJA_ERR_INVALID_ARGUMENT, "backmap_into: bad shape");
  if (!T || !shift || !Y || !V) return fail(NAJA_ERR_INVALID_ARGUMENT, "backmap_into: null argument");
  if (ldt < n) return fail(NAJA_ERR_INVALID_ARGUMENT, "backmap_into: transformation shape mismatch with samples");
  if ((y_dtype != NAJA_DTYPE_F32 && y_dtype != NAJA_DTYPE_F64) || (v_dtype != NAJA_DTYPE_F32 && v_dtype != NAJA_DTYPE_F64))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "backmap_into: unknown dtype");
  if (int st = require_local("backmap_into", {T, shift, Y, V})) return st;
  if (N == 0) return NAJA_OK;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const size_t ybytes = static_cast<size_t>(N) * d * (y_dtype == NAJA_DTYPE_F64 ? 8 : 4);
  const size_t vbytes = static_cast<size_t>(N) * n * (v_dtype == NAJA_DTYPE_F64 ? 8 : 4);
  DeviceBuffer bT, bs, bY, bV;
  const void *dT = nullptr, *dS = nullptr, *dY = nullptr;
  int st;
  if ((st = device_view(T, static_cast<size_t>(ldt) * (d - 1) * 8 + static_cast<size_t>(n) * 8, stream, bT, &dT)))
    return st;
  if ((st = device_view(shift, static_cast<size_t>(n) * 8, stream, bs, &dS))) return st;
  if ((st = device_view(Y, ybytes, stream, bY, &dY))) return st;
  void* dV = V;
  const bool host_v = !is_device_ptr(V);
  if (host_v) {
    if ((st = bV.alloc(vbytes, stream))) return st;
    dV = bV.ptr;
  }
  const double* Td = static_cast<const double*>(dT);
  const double* Sd = static_cast<const double*>(dS);
  if (mode == NAJA_BACKMAP_FP64) {
    if ((st = backmap_fp64_enqueue(n, d, N, Td, ldt, Sd, dY, y_dtype, dV, v_dtype, stream))) return st;
  } else if (mode == NAJA_BACKMAP_BF16X3 || mode == NAJA_BACKMAP_TF32X3) {
    st = backmap_tc(n, d, N, Td, ldt, Sd, dY, y_dtype, dV, v_dtype, mode, stream);
    if (st) return st;
  } else {
    return fail(NAJA_ERR_INVALID_ARGUMENT, "backmap: unknown mode");
  }
  cudaError_t e = cudaSuccess;
  if (host_v) e = cudaMemcpyAsync(V, dV, vbytes, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess && (host_v || bT.ptr || bs.ptr || bY.ptr)) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("backmap: ") + cudaGetErrorString(e));
  return NAJA_OK;
}

extern "C" int naja_backmap_noalloc(int n, int d, long long N, const double* T, int ldt, const double* shift,
                                    const void* Y, int y_dtype, void* V, int v_dtype, int mode, void* stream_ptr) {
  if (n <= 0 || d <= 0 || N < 0) return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_backmap_noalloc: bad shape");
  if (!T || !shift || !Y || !V) return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_backmap_noalloc: null argument");
  if (ldt < n) return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_backmap_noalloc: ldt < n");
  if ((y_dtype != NAJA_DTYPE_F32 && y_dtype != NAJA_DTYPE_F64) || (v_dtype != NAJA_DTYPE_F32 && v_dtype != NAJA_DTYPE_F64))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_backmap_noalloc: unknown dtype");
  if (mode != NAJA_BACKMAP_BF16X3 && mode != NAJA_BACKMAP_TF32X3)
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_backmap_noalloc: mode must be NAJA_BACKMAP_BF16X3 or NAJA_BACKMAP_TF32X3");
  // Host buffers would need staging copies, i.e. allocations: every buffer must be device memory.
  if (!is_device_ptr(T) || !is_device_ptr(shift) || !is_device_ptr(Y) || !is_device_ptr(V))
    return fail(NAJA_ERR_INVALID_ARGUMENT, "naja_backmap_noalloc: T, shift, Y and V must be device memory");
  if (int st = require_local("naja_backmap_noalloc", {T, shift, Y, V})) return st;
  if (N == 0) return NAJA_OK;
  return backmap_tc_noalloc(n, d, N, T, ldt, shift, Y, y_dtype, V, v_dtype, mode, static_cast<cudaStream_t>(stream_ptr));
}
