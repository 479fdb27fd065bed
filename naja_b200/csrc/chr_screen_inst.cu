// One (element type, consumer thread count) slice of the screened CHR
// kernel's instantiations, compiled as its own translation unit so that the
// build runs in parallel.  NAJA_CHR_REAL and NAJA_CHR_NT are set by the build.
#include "chr_screen.cuh"

#define NAJA_CAT3_(a, b, c) a##_##b##_##c
#define NAJA_CAT3(a, b, c) NAJA_CAT3_(a, b, c)

namespace naja {
// cfg.rows = chunks of every warp
int NAJA_CAT3(chr_screen_launch, NAJA_CHR_REAL, NAJA_CHR_NT)(const ChrArgs& a, int nchains, const ChrLaunchConfig& cfg,
                                                            cudaStream_t stream) {
  using namespace chr_detail;
  using Real = NAJA_CHR_REAL;
  constexpr int NT = NAJA_CHR_NT;
#define NAJA_SCREEN_CASE(R)                                    \
  case R:                                                      \
    if constexpr (R <= screen_max_chunks(sizeof(Real) == 8, NT)) \
      return launch_screen<Real, NT, R>(a, nchains, cfg, stream); \
    break;
  switch (cfg.rows) {
    NAJA_SCREEN_CASE(1)
    NAJA_SCREEN_CASE(2)
    NAJA_SCREEN_CASE(3)
    NAJA_SCREEN_CASE(4)
    NAJA_SCREEN_CASE(5)
    NAJA_SCREEN_CASE(6)
    NAJA_SCREEN_CASE(7)
    NAJA_SCREEN_CASE(8)
    default: break;
  }
#undef NAJA_SCREEN_CASE
  return NAJA_ERR_UNSUPPORTED;
}
}  // namespace naja
