// One consumer-thread-count slice of the batched CHR kernel's instantiations
// (NAJA_CHR_NT is set by the build).
#include "chr_batched.cuh"
#include "chr_screen.cuh"

#define NAJA_CAT2_(a, b) a##_##b
#define NAJA_CAT2(a, b) NAJA_CAT2_(a, b)

namespace naja {
int NAJA_CAT2(chr_batch_dispatch, NAJA_CHR_NT)(const ChrArgs* base, const ModelDesc* models, const int* im,
                                              const int* ic, int nitems, const BatchConfig& cfg, cudaStream_t stream,
                                              int* occ_out) {
  if (cfg.screen) {
    using chr_detail::batch_screen_one;
    switch (cfg.rows) {
      case 1: return batch_screen_one<NAJA_CHR_NT, 1>(base, models, im, ic, nitems, cfg, stream, occ_out);
      case 2: return batch_screen_one<NAJA_CHR_NT, 2>(base, models, im, ic, nitems, cfg, stream, occ_out);
      case 3: return batch_screen_one<NAJA_CHR_NT, 3>(base, models, im, ic, nitems, cfg, stream, occ_out);
      case 4: return batch_screen_one<NAJA_CHR_NT, 4>(base, models, im, ic, nitems, cfg, stream, occ_out);
      case 5: return batch_screen_one<NAJA_CHR_NT, 5>(base, models, im, ic, nitems, cfg, stream, occ_out);
      case 6: return batch_screen_one<NAJA_CHR_NT, 6>(base, models, im, ic, nitems, cfg, stream, occ_out);
      default: return NAJA_ERR_UNSUPPORTED;
    }
  }
  return chr_detail::batch_dispatch<NAJA_CHR_NT>(base, models, im, ic, nitems, cfg, stream, occ_out);
}
}  // namespace naja
