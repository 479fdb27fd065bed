// Split-precision tensor-core backmap V = Y T^T + shift on sm_100a (tcgen05).
//
// GEMM view: D (M x N) = A (M x K) B (N x K)^T with A = samples Y (K-major,
// one row per sample), B = T (K-major after a transpose), K = d.  FP32 values
// are carried by two lower-precision terms, x = hi + lo, and the product is
// taken as hi*hi + hi*lo + lo*hi (the lo*lo term is below the terms' own
// rounding), accumulated in FP32 in tensor memory:
//   BF16X3 : hi = bf16(x), lo = bf16(x - hi)            (kind::f16, BF16 in)
//   TF32X3 : hi = tf32(x), lo = tf32(x - hi)            (kind::tf32)
//
// Organisation (a cluster of two CTAs per pair of SMs, persistent over 256 x
// 256 output tiles, tiles ordered n-fastest so a sample block stays in L2
// across its n tiles).  CTA r of a pair holds rows 128 r .. 128 r + 127 of the
// samples and of the outputs; the pair's tensor cores take both halves of B
// (tcgen05.mma cta_group::2), so each SM stages and reads half of it.  What
// bounds a single CTA's 128 x 256 tile is shared memory: 96 KB written and
// twelve products of 12 KB read per slice, 1,920 cycles at 128 bytes a clock
// against 1,536 of the tensor core; a pair's CTA writes 64 KB and reads 8 KB
// per product, 1,280.
//   warp 4, one thread : TMA producer of its CTA.  2-D tiled bulk-tensor loads
//                        with 128-byte swizzle of its halves of A_hi, A_lo,
//                        B_hi, B_lo for one 128-byte K slice into a 3-stage
//                        shared-memory ring; they complete on the first CTA's
//                        barrier.
//   warp 5, one thread of the first CTA : MMA issuer.  Per stage 4 K-steps x 3
//                        tcgen05.mma into one of two 256-column FP32
//                        accumulators in each CTA's TMEM (512 columns; tiles
//                        alternate), so a tile's MMAs run while the epilogue
//                        drains the previous tile; tcgen05.commit releases
//                        the stage in both CTAs.
//   warps 0-3          : epilogue of their CTA's 128 rows.  tcgen05.ld of their
//                        32 TMEM lanes, 32 x 32 blocks transposed through
//                        shared memory, + shift, stores of 32 consecutive
//                        values of a row each.
// N 50,001, n 2,600, d 700, TF32X3: GEMM 1,080 -> 847 us; N 30,011, n 6,999,
// d 1,501, BF16X3: 1,716 -> 1,388 us.
// Every wait is bounded (global timer); on expiry the CTA records an error,
// stops issuing, drains the pair's copies / MMAs and frees TMEM; the pair leaves
// together.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/naja_chr.h"
#include "capi_internal.cuh"
#include "common.cuh"

namespace naja {
namespace {

constexpr int kCtaM = 128;           // rows of A of a CTA
constexpr int kTileM = 2 * kCtaM;    // of a pair
constexpr int kTileN = 256;
constexpr int kCtaN = kTileN / 2;    // rows of B that a CTA stages
constexpr int kSliceBytes = 128;  // K extent of one stage, in bytes per row
constexpr int kStages = 3;
constexpr int kThreads = 192;     // warps 0-3 epilogue, 4 producer, 5 MMA
constexpr uint32_t kTmemCols = 512;  // two 256-column accumulators
constexpr uint64_t kTimeoutNs = 5ull * 1000 * 1000 * 1000;

constexpr uint32_t kATileBytes = kCtaM * kSliceBytes;  // 16 KB
constexpr uint32_t kBTileBytes = kCtaN * kSliceBytes;  // 16 KB
constexpr uint32_t kStageBytes = 2 * kATileBytes + 2 * kBTileBytes;

enum TcError : int { kTcTimeoutLoad = 11, kTcTimeoutSlot = 12, kTcTimeoutAcc = 13, kTcTimeoutEpi = 14 };

struct TcArgs {
  int n, kslices;
  long long N;
  int tiles_n;
  long long tiles;
  const double* shift;
  void* V;
  int v_f64;
  int* err;
};

// ------------------------------------------------------------ PTX wrappers
// Completes on the barrier at a shared::cluster address, this CTA's or its
// pair's.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// K-major, 128-byte-swizzled operand: 8-row core groups 1024 B apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(const void* smem) {
  const uint64_t addr = smem_u32(smem);
  uint64_t d = 0;
  d |= (addr >> 4) & 0x3FFFull;              // start address
  d |= static_cast<uint64_t>(1) << 16;        // leading byte offset (unused with swizzle)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;  // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;        // descriptor version (sm100)
  d |= static_cast<uint64_t>(2) << 61;        // SWIZZLE_128B
  return d;
}

template <bool TF32>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  if constexpr (TF32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
  }
}

// Arrives on the barrier at this offset in both CTAs once the MMAs issued so
// far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ------------------------------------------------------------------ kernel
template <bool TF32>
__global__ void __launch_bounds__(kThreads, 1)
    backmap_tc_kernel(const __grid_constant__ CUtensorMap mAhi, const __grid_constant__ CUtensorMap mAlo,
                      const __grid_constant__ CUtensorMap mBhi, const __grid_constant__ CUtensorMap mBlo, TcArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte alignment for the swizzled tiles
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;  // [2]
  uint64_t* acc_empty = acc_full + 2;    // [2]
  uint64_t* drain_bar = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // epilogue staging: one 32 x 33 float block per epilogue warp
  float* stage_out = reinterpret_cast<float*>(smem + kStages * kStageBytes + 256);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&acc_full[0], 1);
    mbar_init(&acc_full[1], 1);
    mbar_init(&acc_empty[0], 8);  // the epilogue warps of both CTAs
    mbar_init(&acc_empty[1], 8);
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers and TMEM are there
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t rank = cluster_rank();
  const long long pair = blockIdx.x / 2, pairs = gridDim.x / 2;

  const int K = a.kslices;
  if (warp == 4) {
    if (lane == 0) {
      // ---------------- TMA producer
      int stage = 0;
      uint32_t round = 0;
      uint32_t last_parity = 0, used = 0;
      const int elem_per_slice = TF32 ? 32 : 64;
      for (long long tile = pair; tile < a.tiles && !*abort_flag; tile += pairs) {
        const int tm = static_cast<int>(tile / a.tiles_n), tn = static_cast<int>(tile % a.tiles_n);
        for (int ks = 0; ks < K; ++ks) {
          if (round >= 1 && !mbar_wait_bounded(&empty[stage], (round - 1) & 1u, kTimeoutNs)) {
            set_error(a.err, kTcTimeoutSlot, static_cast<int>(blockIdx.x), stage, ks);
            *abort_flag = 1;
            break;
          }
          unsigned char* st = smem + stage * kStageBytes;
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * kStageBytes);  // both CTAs' loads
          const int x = ks * elem_per_slice, ya = tm * kTileM + static_cast<int>(rank) * kCtaM,
                    yb = tn * kTileN + static_cast<int>(rank) * kCtaN;
          const uint32_t bar = cluster_map(&full[stage], 0);
          tma_load_2d_pair(st, &mAhi, x, ya, bar);
          tma_load_2d_pair(st + kATileBytes, &mAlo, x, ya, bar);
          tma_load_2d_pair(st + 2 * kATileBytes, &mBhi, x, yb, bar);
          tma_load_2d_pair(st + 2 * kATileBytes + kBTileBytes, &mBlo, x, yb, bar);
          used |= 1u << stage;
          last_parity = (last_parity & ~(1u << stage)) | ((round & 1u) << stage);
          if (++stage == kStages) {
            stage = 0;
            ++round;
          }
        }
      }
      // drain: every issued load of the pair has landed before it may exit
      for (int s = 0; s < kStages && rank == 0; ++s)
        if (((used >> s) & 1u) && !mbar_wait_bounded(&full[s], (last_parity >> s) & 1u, kTimeoutNs))
          set_error(a.err, kTcTimeoutLoad, static_cast<int>(blockIdx.x), s, -1);
    }
  } else if (warp == 5) {
    if (lane == 0 && rank == 0) {
      // ---------------- MMA issuer
      constexpr uint32_t fmt = TF32 ? 2u : 1u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(kTileN >> 3) << 17) |
                             (static_cast<uint32_t>(kTileM >> 4) << 24);
      constexpr int ksteps = 4;             // 4 MMAs of 32 bytes of K per 128-byte slice
      int stage = 0;
      uint32_t parity = 0;
      uint32_t acc_round = 0;  // tiles issued by this CTA; accumulator acc_round & 1
      bool issued = false;
      for (long long tile = pair; tile < a.tiles && !*abort_flag; tile += pairs) {
        const uint32_t buf = acc_round & 1u, use = acc_round >> 1;
        const uint32_t tacc = tmem + buf * static_cast<uint32_t>(kTileN);
        // the epilogue has read this accumulator's previous tile (two tiles back)
        if (use >= 1 && !mbar_wait_cluster_bounded(&acc_empty[buf], (use - 1) & 1u, kTimeoutNs)) {
          set_error(a.err, kTcTimeoutEpi, static_cast<int>(blockIdx.x), static_cast<int>(acc_round), -1);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        bool ok = true;
        for (int ks = 0; ks < K; ++ks) {
          if (!mbar_wait_cluster_bounded(&full[stage], parity, kTimeoutNs)) {
            set_error(a.err, kTcTimeoutLoad, static_cast<int>(blockIdx.x), stage, ks);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          unsigned char* st = smem + stage * kStageBytes;
          const unsigned char* Ahi = st;
          const unsigned char* Alo = st + kATileBytes;
          const unsigned char* Bhi = st + 2 * kATileBytes;
          const unsigned char* Blo = st + 2 * kATileBytes + kBTileBytes;
#pragma unroll
          for (int kk = 0; kk < ksteps; ++kk) {
            const uint64_t ah = umma_desc_sw128(Ahi + kk * 32), al = umma_desc_sw128(Alo + kk * 32);
            const uint64_t bh = umma_desc_sw128(Bhi + kk * 32), bl = umma_desc_sw128(Blo + kk * 32);
            const uint32_t acc = (ks > 0 || kk > 0) ? 1u : 0u;
            umma<TF32>(tacc, ah, bh, idesc, acc);
            umma<TF32>(tacc, ah, bl, idesc, 1u);
            umma<TF32>(tacc, al, bh, idesc, 1u);
          }
          issued = true;
          umma_commit_pair(&empty[stage]);  // the stage is free once these MMAs have read it
          if (++stage == kStages) {
            stage = 0;
            parity ^= 1u;
          }
        }
        if (!ok) break;
        umma_commit_pair(&acc_full[buf]);  // accumulator complete
        ++acc_round;
      }
      if (issued) {
        // every MMA of this CTA has finished before TMEM is released
        umma_commit_pair(drain_bar);
        if (!mbar_wait_bounded(drain_bar, 0u, kTimeoutNs)) set_error(a.err, kTcTimeoutAcc, static_cast<int>(blockIdx.x), -1, -1);
      }
    }
  } else {
    // ---------------- epilogue, warps 0-3: TMEM lanes 32*warp .. 32*warp+31
    // Each 32 x 32 block goes through shared memory so that every store
    // instruction writes 32 consecutive values of one output row.  The
    // other accumulator takes the next tile's MMAs meanwhile.
    float* stg = stage_out + warp * (32 * 33);
    uint32_t acc_round = 0;
    for (long long tile = pair; tile < a.tiles; tile += pairs) {
      const uint32_t buf = acc_round & 1u, use = acc_round >> 1;
      bool ok = mbar_wait_bounded(&acc_full[buf], use & 1u, kTimeoutNs);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) set_error(a.err, kTcTimeoutAcc, static_cast<int>(blockIdx.x), warp, static_cast<int>(acc_round));
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      const int tm = static_cast<int>(tile / a.tiles_n), tn = static_cast<int>(tile % a.tiles_n);
      const long long row_base = static_cast<long long>(tm) * kTileM + static_cast<int>(rank) * kCtaM + warp * 32;
      const int col0 = tn * kTileN;
#pragma unroll 1
      for (int c = 0; c < kTileN; c += 32) {
        uint32_t r[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + buf * static_cast<uint32_t>(kTileN) +
                      static_cast<uint32_t>(c),
                  r);
#pragma unroll
        for (int q = 0; q < 32; ++q) stg[lane * 33 + q] = __uint_as_float(r[q]);
        __syncwarp();
        const int i = col0 + c + lane;
        const bool col_ok = i < a.n;
        const double sh = col_ok ? a.shift[i] : 0.0;
        // eight rows at a time, their conversions and stores independent of
        // one another (a row's chain of read, conversion, FP64 addition,
        // conversion and store is some 200 cycles: one row after another, a
        // tile's epilogue took twice as long as its products)
        const int rows = a.N - row_base < 32 ? static_cast<int>(a.N - row_base) : 32;
        auto put = [&](auto* v) {
          using VT = typename std::remove_pointer<decltype(v)>::type;
          v += row_base * a.n + i;
          int j = 0;
          if (col_ok) {
            for (; j + 8 <= rows; j += 8) {
              VT o[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) o[u] = static_cast<VT>(static_cast<double>(stg[(j + u) * 33 + lane]) + sh);
#pragma unroll
              for (int u = 0; u < 8; ++u) v[static_cast<long long>(j + u) * a.n] = o[u];
            }
            for (; j < rows; ++j)
              v[static_cast<long long>(j) * a.n] = static_cast<VT>(static_cast<double>(stg[j * 33 + lane]) + sh);
          }
        };
        if (a.v_f64) put(reinterpret_cast<double*>(a.V));
        else put(reinterpret_cast<float*>(a.V));
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(cluster_map(&acc_empty[buf], 0));
      ++acc_round;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA's memory or TMEM is in use any more
  tc_fence_after();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ----------------------------------------------------------- operand split
// Y (N x d, row-major, float or double) -> hi, lo (N x dp, row-major), zero
// for k >= d.  T (n x d column-major, ldt) -> hi, lo (n x dp row-major).
// Both are bound by memory; one warp per row and 16-byte pieces (Y), 32 x 32
// blocks through shared memory (T, whose columns are contiguous where its
// split rows are): 50,001 x 700 samples 106 -> 66 us, T 6,999 x 1,501
// 52 -> 21 us.
template <bool TF32>
__device__ __forceinline__ void split_value(float x, uint32_t& hi, uint32_t& lo) {
  if constexpr (TF32) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
  } else {
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
    hi = __bfloat16_as_ushort(h);
    lo = __bfloat16_as_ushort(l);
  }
}

// Four consecutive split values at element `at` (a multiple of 4).
template <bool TF32>
__device__ __forceinline__ void split_store(void* dst, long long at, const uint32_t (&v)[4]) {
  if constexpr (TF32)
    *reinterpret_cast<uint4*>(static_cast<uint32_t*>(dst) + at) = make_uint4(v[0], v[1], v[2], v[3]);
  else
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(dst) + at) = make_uint2(v[0] | v[1] << 16, v[2] | v[3] << 16);
}

// WIDE: rows of Y start on 16 bytes and d is a multiple of 4.
template <class YT, bool TF32, bool WIDE>
__global__ void __launch_bounds__(256) split_rows_kernel(const YT* __restrict__ Y, long long N, int d, int dp, void* hi,
                                                         void* lo) {
  const int lane = threadIdx.x & 31;
  for (long long s = blockIdx.x * 8LL + (threadIdx.x >> 5); s < N; s += gridDim.x * 8LL) {
    const YT* y = Y + s * d;
    for (int k = lane * 4; k < dp; k += 128) {
      float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if constexpr (WIDE) {
        if (k < d) {
          if constexpr (sizeof(YT) == 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(y + k));
            x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
          } else {
            const double2 v = __ldg(reinterpret_cast<const double2*>(y + k)), w = __ldg(reinterpret_cast<const double2*>(y + k + 2));
            x[0] = static_cast<float>(v.x), x[1] = static_cast<float>(v.y);
            x[2] = static_cast<float>(w.x), x[3] = static_cast<float>(w.y);
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (k + q < d) x[q] = static_cast<float>(y[k + q]);
      }
      uint32_t h[4], l[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) split_value<TF32>(x[q], h[q], l[q]);
      split_store<TF32>(hi, s * dp + k, h);
      split_store<TF32>(lo, s * dp + k, l);
    }
  }
}

// 256 threads, 32 rows (outputs) x 32 columns of T per block.
template <bool TF32>
__global__ void __launch_bounds__(256) split_T_kernel(const double* __restrict__ T, int ldt, int n, int d, int dp, void* hi,
                                                      void* lo) {
  __shared__ float t[32][33];
  const int i0 = blockIdx.x * 32, k0 = blockIdx.y * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
  for (int q = y; q < 32; q += 8)
    t[x][q] = i0 + x < n && k0 + q < d ? static_cast<float>(T[static_cast<long long>(k0 + q) * ldt + i0 + x]) : 0.0f;
  __syncthreads();
  const int i = threadIdx.x >> 3, k = threadIdx.x % 8 * 4;
  if (i0 + i < n) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) split_value<TF32>(t[i][k + q], h[q], l[q]);
    split_store<TF32>(hi, static_cast<long long>(i0 + i) * dp + k0 + k, h);
    split_store<TF32>(lo, static_cast<long long>(i0 + i) * dp + k0 + k, l);
  }
}

// ------------------------------------------------------------ tensor maps
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// 2-D map over a row-major rows x dp matrix; box = box_rows x (128 bytes).
bool make_map(CUtensorMap* m, void* base, bool tf32, long long rows, int dp, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return false;
  const CUtensorMapDataType dt = tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int esz = tf32 ? 4 : 2;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(dp), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(dp) * esz};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(kSliceBytes / esz), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, dt, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace

size_t backmap_tc_operand_bytes(long long rows, int d, int mode) {
  const size_t esz = mode == NAJA_BACKMAP_TF32X3 ? 4 : 2;
  const size_t dp = static_cast<size_t>((d + 63) / 64 * 64);
  return (static_cast<size_t>(rows) * dp * esz + 1023) / 1024 * 1024;
}

int backmap_tc_split_T(int n, int d, const double* T, int ldt, void* Th, void* Tl, int mode, cudaStream_t stream) {
  const int dp = (d + 63) / 64 * 64;
  const dim3 grid((n + 31) / 32, dp / 32);
  if (mode == NAJA_BACKMAP_TF32X3)
    split_T_kernel<true><<<grid, 256, 0, stream>>>(T, ldt, n, d, dp, Th, Tl);
  else
    split_T_kernel<false><<<grid, 256, 0, stream>>>(T, ldt, n, d, dp, Th, Tl);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("backmap: split launch failed: ") + cudaGetErrorString(e));
  return NAJA_OK;
}

namespace {
int enqueue_rows(int n, int d, long long N, const void* Y, int y_dtype, const void* Th, const void* Tl, void* Yh,
                 void* Yl, const double* shift, void* V, int v_dtype, int mode, int* err, cudaStream_t stream) {
  const bool tf32 = mode == NAJA_BACKMAP_TF32X3;
  const int esz = tf32 ? 4 : 2;
  const int dp = (d + 63) / 64 * 64;
  auto split = [&](auto* y) {
    using YT = typename std::remove_const<typename std::remove_pointer<decltype(y)>::type>::type;
    const bool wide = d % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15u) == 0;
    auto kern = tf32 ? (wide ? split_rows_kernel<YT, true, true> : split_rows_kernel<YT, true, false>)
                     : (wide ? split_rows_kernel<YT, false, true> : split_rows_kernel<YT, false, false>);
    const int blocks = static_cast<int>(std::min<long long>((N + 7) / 8, 148 * 16));
    kern<<<blocks, 256, 0, stream>>>(y, N, d, dp, Yh, Yl);
  };
  if (y_dtype == NAJA_DTYPE_F64) split(static_cast<const double*>(Y));
  else split(static_cast<const float*>(Y));
  CUtensorMap mAh, mAl, mBh, mBl;
  if (!make_map(&mAh, Yh, tf32, N, dp, kCtaM) || !make_map(&mAl, Yl, tf32, N, dp, kCtaM) ||
      !make_map(&mBh, const_cast<void*>(Th), tf32, n, dp, kCtaN) ||
      !make_map(&mBl, const_cast<void*>(Tl), tf32, n, dp, kCtaN))
    return fail(NAJA_ERR_CUDA, "backmap: cuTensorMapEncodeTiled failed");
  TcArgs a;
  a.n = n;
  a.kslices = dp * esz / kSliceBytes;
  a.N = N;
  a.tiles_n = (n + kTileN - 1) / kTileN;
  a.tiles = ((N + kTileM - 1) / kTileM) * a.tiles_n;
  a.shift = shift;
  a.V = V;
  a.v_f64 = v_dtype == NAJA_DTYPE_F64;
  a.err = err;
  const size_t smem = kStages * kStageBytes + 1024 + 256 + 4 * 32 * 33 * sizeof(float);
  int sms = 148, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = 2 * static_cast<int>(std::min<long long>(sms / 2, a.tiles));
  auto kern = tf32 ? backmap_tc_kernel<true> : backmap_tc_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("backmap: ") + cudaGetErrorString(e));
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(static_cast<unsigned>(grid));
  lc.blockDim = dim3(kThreads);
  lc.dynamicSmemBytes = smem;
  lc.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  e = cudaLaunchKernelEx(&lc, kern, mAh, mAl, mBh, mBl, a);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("backmap: launch failed: ") + cudaGetErrorString(e));
  return NAJA_OK;
}

}  // namespace

// Samples that naja_backmap splits and maps at a time (the overlapped pipeline
// maps a chunk of its chains at one go): the split operands of a chunk stay in L2
// between the kernel that writes them and the GEMM that reads them (about 112
// MB beside T's), a call's scratch does not grow with its samples, and the
// chunk's tiles fill whole rounds of the pairs of SMs as well as any number of
// row blocks near that size can.
long long backmap_tc_chunk_rows(long long N, int n, int d, int mode) {
  const long long row_bytes = 2LL * ((d + 63) / 64 * 64) * (mode == NAJA_BACKMAP_TF32X3 ? 4 : 2);
  const long long most = std::max(1LL, (112LL << 20) / (row_bytes * kTileM));  // row blocks
  if (N <= most * kTileM) return N;
  const long long tiles_n = (n + kTileN - 1) / kTileN, pairs = 74;
  long long best = most;
  double best_use = 0.0;
  for (long long b = most; 2 * b >= most && b >= 1; --b) {
    const long long rounds = (b * tiles_n + pairs - 1) / pairs;
    const double use = static_cast<double>(b * tiles_n) / static_cast<double>(rounds * pairs);
    if (use > best_use + 1e-9) {
      best_use = use;
      best = b;
    }
  }
  return best * kTileM;
}

int backmap_tc_enqueue(int n, int d, long long N, long long chunk, const void* Y, int y_dtype, const void* Th,
                       const void* Tl, void* Yh, void* Yl, const double* shift, void* V, int v_dtype, int mode, int* err,
                       cudaStream_t stream) {
  const size_t ys = y_dtype == NAJA_DTYPE_F64 ? 8 : 4, vs = v_dtype == NAJA_DTYPE_F64 ? 8 : 4;
  for (long long r = 0; r < N; r += chunk) {
    const int st = enqueue_rows(n, d, std::min(chunk, N - r), static_cast<const char*>(Y) + r * d * ys, y_dtype, Th, Tl,
                                Yh, Yl, shift, static_cast<char*>(V) + r * n * vs, v_dtype, mode, err, stream);
    if (st) return st;
  }
  return NAJA_OK;
}

int backmap_tc_read_error(const int* err, cudaStream_t stream, const char* who) {
  int w[4] = {0, 0, 0, 0};
  cudaError_t e = cudaMemcpyAsync(w, err, sizeof(w), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string(who) + ": " + cudaGetErrorString(e));
  if (w[0] != 0)
    return fail(NAJA_ERR_DEVICE, std::string(who) + ": tensor-core pipeline gave up a bounded wait (code " +
                                     std::to_string(w[0]) + ", " + std::to_string(w[1]) + ", " + std::to_string(w[2]) +
                                     ", " + std::to_string(w[3]) + ")");
  return NAJA_OK;
}

int backmap_tc(int n, int d, long long N, const double* T, int ldt, const double* shift, const void* Y, int y_dtype,
               void* V, int v_dtype, int mode, cudaStream_t stream) {
  const long long chunk = backmap_tc_chunk_rows(N, n, d, mode);
  const size_t ybytes = backmap_tc_operand_bytes(chunk, d, mode), tbytes = backmap_tc_operand_bytes(n, d, mode);
  DeviceBuffer bYh, bYl, bTh, bTl, berr;
  int st;
  if ((st = bYh.alloc(ybytes, stream)) || (st = bYl.alloc(ybytes, stream)) || (st = bTh.alloc(tbytes, stream)) ||
      (st = bTl.alloc(tbytes, stream)) || (st = berr.alloc(4 * sizeof(int), stream)))
    return st;
  int* err = static_cast<int*>(berr.ptr);
  cudaError_t e = cudaMemsetAsync(err, 0, 4 * sizeof(int), stream);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("backmap: ") + cudaGetErrorString(e));
  if ((st = backmap_tc_split_T(n, d, T, ldt, bTh.ptr, bTl.ptr, mode, stream))) return st;
  if ((st = backmap_tc_enqueue(n, d, N, chunk, Y, y_dtype, bTh.ptr, bTl.ptr, bYh.ptr, bYl.ptr, shift, V, v_dtype, mode, err,
                               stream)))
    return st;
  return backmap_tc_read_error(err, stream, "backmap");
}

// ----------------------------------------------------------------------
// Allocation-free variant (naja_backmap_noalloc).
//
// Some callers cannot allocate device memory at the point they need the
// backmap: a service that reserves its whole device-memory budget up front
// and forbids allocations in its request path, or a host framework whose
// allocator owns the device and must not see cudaMalloc/cudaFree (which may
// also synchronise the device) from a library.  For them the split operands
// live in one file-scope device array of fixed size instead of per-call
// buffers.  The array exists once per device that loads this library and is
// held until the process exits.  Its device address is looked up once per
// device (cudaGetSymbolAddress, with that device current) on the first call
// made on that device; that first call should therefore come before any
// stream capture.  After cudaDeviceReset the cached address is stale: a
// process that resets a device must not call this entry point on it again.
// Every call reuses the same array: the error words are cleared by each call,
// and calls whose work overlaps on the GPU (different streams, or different
// host threads on one device) race on the array, so the caller serialises
// them.
constexpr size_t kNoAllocScratchBytes = 64ull << 20;  // 64 MiB
constexpr int kNoAllocMaxDevices = 64;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace {
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kNoAllocMaxDevices] = {};

int noalloc_scratch(unsigned char** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("naja_backmap_noalloc: ") + cudaGetErrorString(e));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(NAJA_ERR_UNSUPPORTED, "naja_backmap_noalloc: device index too large");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      return fail(NAJA_ERR_CUDA, std::string("naja_backmap_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return NAJA_OK;
}
}  // namespace

int backmap_tc_noalloc(int n, int d, long long N, const double* T, int ldt, const double* shift, const void* Y,
                       int y_dtype, void* V, int v_dtype, int mode, cudaStream_t stream) {
  // scratch layout: [error words | Y hi | Y lo | T hi | T lo], each 1024-aligned
  const size_t ybytes = backmap_tc_operand_bytes(N, d, mode), tbytes = backmap_tc_operand_bytes(n, d, mode);
  const size_t need = 1024 + 2 * ybytes + 2 * tbytes;
  if (need > kNoAllocScratchBytes)
    return fail(NAJA_ERR_INVALID_ARGUMENT,
                "naja_backmap_noalloc: this shape needs " + std::to_string(need) + " bytes of scratch, more than the " +
                    std::to_string(kNoAllocScratchBytes) + " the library reserves; pass fewer samples per call");
  unsigned char* base = nullptr;
  int st = noalloc_scratch(&base);
  if (st) return st;
  int* err = reinterpret_cast<int*>(base);
  void* Yh = base + 1024;
  void* Yl = base + 1024 + ybytes;
  void* Th = base + 1024 + 2 * ybytes;
  void* Tl = base + 1024 + 2 * ybytes + tbytes;
  cudaError_t e = cudaMemsetAsync(err, 0, 4 * sizeof(int), stream);
  if (e != cudaSuccess) return fail(NAJA_ERR_CUDA, std::string("naja_backmap_noalloc: ") + cudaGetErrorString(e));
  if ((st = backmap_tc_split_T(n, d, T, ldt, Th, Tl, mode, stream))) return st;
  if ((st = backmap_tc_enqueue(n, d, N, N, Y, y_dtype, Th, Tl, Yh, Yl, shift, V, v_dtype, mode, err, stream))) return st;
  return backmap_tc_read_error(err, stream, "naja_backmap_noalloc");
}

}  // namespace naja
