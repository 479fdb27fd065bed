// One row-warp-count slice of the batched private-rows compressed-column
// kernel's instantiations (NAJA_CHR_NW is set by the build).
#include "chr_columns.cuh"

#define NAJA_CAT2_(a, b) a##_##b
#define NAJA_CAT2(a, b) NAJA_CAT2_(a, b)

namespace naja {
int NAJA_CAT2(chr_columns_batch, NAJA_CHR_NW)(const ChrArgs* base, const ModelDesc* models, const int* im,
                                             const int* ic, int nitems, const BatchConfig& cfg, cudaStream_t stream,
                                             int* occ_out) {
  using chr_detail::batch_columns_one;
  constexpr int NW = NAJA_CHR_NW;
  switch (cfg.entries) {
    case 1: return batch_columns_one<NW, 1>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 2: return batch_columns_one<NW, 2>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 3: return batch_columns_one<NW, 3>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 4: return batch_columns_one<NW, 4>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 5: return batch_columns_one<NW, 5>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 6: return batch_columns_one<NW, 6>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 8: return batch_columns_one<NW, 8>(base, models, im, ic, nitems, cfg, stream, occ_out);
    default: return NAJA_ERR_UNSUPPORTED;
  }
}
}  // namespace naja
