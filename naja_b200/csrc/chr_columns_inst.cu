// One (element type, row warps) slice of the private-rows compressed-column
// kernel's instantiations (NAJA_CHR_REAL and NAJA_CHR_NW are set by the build).
#include "chr_columns.cuh"

#define NAJA_CAT3_(a, b, c) a##_##b##_##c
#define NAJA_CAT3(a, b, c) NAJA_CAT3_(a, b, c)

namespace naja {
namespace chr_detail {
namespace {
template <class Real, int NW, int E, bool RES>
int launch_columns(const ChrArgs& a, const SpArgs& sp, int nchains, const ChrLaunchConfig& cfg, cudaStream_t stream) {
  auto kern = chr_columns_kernel<Real, NW, E, RES>;
  cudaError_t e = allow_smem(kern);
  if (e != cudaSuccess) return NAJA_ERR_CUDA;
  const ColLayout L = make_col_layout(a.d, a.m, sizeof(Real), NW, E, cfg.resident ? 0 : cfg.slots);
  kern<<<nchains, NW * 32 + 64, cfg.smem, stream>>>(a, sp, L);
  return cudaGetLastError() == cudaSuccess ? NAJA_OK : NAJA_ERR_CUDA;
}
}  // namespace
}  // namespace chr_detail

int NAJA_CAT3(chr_columns_launch, NAJA_CHR_REAL, NAJA_CHR_NW)(const ChrArgs& a, const SpArgs& sp, int nchains,
                                                             const ChrLaunchConfig& cfg, cudaStream_t stream) {
  using namespace chr_detail;
  constexpr int NW = NAJA_CHR_NW;
#define NAJA_COL_CASE(E)                                                                            \
  case E:                                                                                           \
    if constexpr (NW <= 2)                                                                          \
      if (cfg.resident) return launch_columns<NAJA_CHR_REAL, NW, E, true>(a, sp, nchains, cfg, stream); \
    return launch_columns<NAJA_CHR_REAL, NW, E, false>(a, sp, nchains, cfg, stream);
  switch (cfg.entries) {
    NAJA_COL_CASE(1)
    NAJA_COL_CASE(2)
    NAJA_COL_CASE(3)
    NAJA_COL_CASE(4)
    NAJA_COL_CASE(5)
    NAJA_COL_CASE(6)
    NAJA_COL_CASE(8)
    default: return NAJA_ERR_UNSUPPORTED;
  }
#undef NAJA_COL_CASE
}
}  // namespace naja
