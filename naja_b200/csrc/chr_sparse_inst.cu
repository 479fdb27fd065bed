// Planning and launch of the sparse-column CHR step kernel (chr_sparse.cuh).
#include "chr_columns.cuh"

namespace naja {
#define NAJA_COL_EACH(X) X(1) X(2) X(4) X(8)
#define NAJA_COL_DECL(NW)                                                                                  \
  int chr_columns_launch_float_##NW(const ChrArgs& a, const SpArgs& sp, int nchains, const ChrLaunchConfig& cfg, \
                                    cudaStream_t stream);                                                  \
  int chr_columns_launch_double_##NW(const ChrArgs& a, const SpArgs& sp, int nchains, const ChrLaunchConfig& cfg, \
                                     cudaStream_t stream);
NAJA_COL_EACH(NAJA_COL_DECL)
#undef NAJA_COL_DECL

using namespace chr_detail;

int chr_columns_warps(double mean_col, int tpb) {
  if (tpb > 0) return tpb == 32 || tpb == 64 || tpb == 128 || tpb == 256 ? tpb / 32 : 0;
  // at most two entries of a mean column per lane (us per step, 16 chains,
  // FP32 / FP64: 416 entries per column 0.814 / 1.288 with 8 warps, 0.858 /
  // 1.755 with 4, 0.917 / 2.006 with 2; 200 entries 0.654 / 1.061 with 4; 2
  // entries 0.388 with 1, 0.546 with 4)
  int nw = 1;
  while (nw < 8 && mean_col > 64.0 * nw) nw *= 2;
  return nw;
}

int chr_columns_plan(int precision, int m, int d, int nw, int entries, int max_slots, int nchains, int sms,
                     ChrLaunchConfig* out) {
  const int elt = precision == NAJA_PREC_FP64 ? 8 : 4;
  auto bytes = [&](int slots) { return make_col_layout(d, m, elt, nw, entries, slots).total; };
  int slots = kMaxSlots;
  if (max_slots > 0 && max_slots < slots) slots = max_slots;
  while (slots >= 3 && bytes(slots) > kSmemBudget) --slots;
  if (slots < 3) return NAJA_ERR_UNSUPPORTED;
  // All columns in shared memory where they fit beside the chain's state and
  // the launch's chains do not take longer for it: the registers let 5 chains
  // (two row warps: 4) run on an SM, not as many copies of the columns may fit,
  // and a step with them there takes about 3/4 of one with staged columns.  ms
  // for 1,000 steps in the unit cube of d = 400, resident / staged: 4 chains
  // FP32 0.42 / 0.54, FP64 0.59 / 0.64; 600 chains 1.27 / 0.70, 2.87 / 0.83; d
  // = 200, 2,400 chains FP32 2.14 / 2.48.
  const int most = nw == 1 ? 5 : 4;
  auto rounds = [&](int q) {
    const int fit = static_cast<int>((kSmemBudget + 1024) / (bytes(q) + 1024)), per = fit < most ? fit : most;
    return (nchains + sms * per - 1) / (sms * per);
  };
  out->resident = nw <= 2 && max_slots <= 0 && bytes(0) <= kSmemBudget && 3 * rounds(0) <= 4 * rounds(slots);
  out->threads = nw * 32;
  out->rows = 0;
  out->slots = slots;
  out->smem = bytes(out->resident ? 0 : slots);
  out->cluster = 1;
  out->slice_lda = 0;
  out->max_col = 0;
  out->columns = 1;
  out->entries = entries;
  out->pair_scatter = 0;
  out->screen = 0;
  out->uniform = 0;
  return NAJA_OK;
}

int chr_sparse_plan(int precision, int m, int d, int max_col, double mean_col, int tpb, int max_slots,
                    ChrLaunchConfig* out) {
  if (max_col <= 0) return NAJA_ERR_UNSUPPORTED;
  int threads;
  if (tpb > 0) {
    if (tpb != 32 && tpb != 64 && tpb != 128 && tpb != 256 && tpb != 512) return NAJA_ERR_UNSUPPORTED;
    threads = tpb;
  } else {
    // at most two entries of a mean column per consumer thread: a step's
    // latency is a chain of shared-memory loads, divisions and barriers, and
    // spreading the entries wider shortens it (m = 5200, 416 entries per
    // column, 16 chains: 1.45 us per step with 256 threads, 2.0 us with 128)
    threads = 32;
    while (threads < 512 && mean_col > 2.0 * threads) threads *= 2;
  }
  const bool f64 = precision == NAJA_PREC_FP64;
  const int elt = f64 ? 8 : 4, eb = f64 ? kSpEntryBytes64 : kSpEntryBytes32;
  const int nw = threads / 32;
  // Pair steps through a scratch column where it fits (fewer instructions per
  // step); otherwise by search (no scratch column, m values less).
  int slots = 0;
  bool scatter = true;
  Layout L;
  for (int sc = 1; sc >= 0 && slots == 0; --sc) {
    int s = kMaxSlots;
    if (max_slots > 0 && max_slots < s) s = max_slots;
    L = make_sparse_layout(d, m, elt, eb, max_col, nw, s, sc != 0);
    while (s > 3 && L.total > kSmemBudget) {
      --s;
      L = make_sparse_layout(d, m, elt, eb, max_col, nw, s, sc != 0);
    }
    if (s >= 3 && L.total <= kSmemBudget) {
      slots = s;
      scatter = sc != 0;
    }
  }
  if (slots == 0) return NAJA_ERR_UNSUPPORTED;
  out->threads = threads;
  out->rows = 0;
  out->slots = slots;
  out->smem = L.total;
  out->cluster = 1;
  out->slice_lda = 0;
  out->max_col = max_col;
  out->columns = 0;
  out->entries = 0;
  out->resident = 0;
  out->pair_scatter = scatter ? 1 : 0;
  out->screen = 0;
  out->uniform = 0;
  return NAJA_OK;
}

int chr_sparse_launch(int precision, const ChrArgs& a, const SpArgs& sp, int nchains, const ChrLaunchConfig& cfg,
                      cudaStream_t stream) {
  if (cfg.columns) {
    const bool f64 = precision == NAJA_PREC_FP64;
#define NAJA_COL_LAUNCH(NW)                                                  \
  case 32 * NW:                                                              \
    return f64 ? chr_columns_launch_double_##NW(a, sp, nchains, cfg, stream) \
               : chr_columns_launch_float_##NW(a, sp, nchains, cfg, stream);
    switch (cfg.threads) {
      NAJA_COL_EACH(NAJA_COL_LAUNCH)
      default: return NAJA_ERR_UNSUPPORTED;
    }
#undef NAJA_COL_LAUNCH
  }
  if (precision == NAJA_PREC_FP64) return launch_sparse_nw<double>(a, sp, nchains, cfg, stream);
  return launch_sparse_nw<float>(a, sp, nchains, cfg, stream);
}

#define NAJA_COLB_EACH(X) X(2) X(4) X(8)
#define NAJA_COLB_DECL(NW)                                                                                     \
  int chr_columns_batch_##NW(const ChrArgs* base, const ModelDesc* models, const int* im, const int* ic, int nitems, \
                             const BatchConfig& cfg, cudaStream_t stream, int* occ_out);
NAJA_COLB_EACH(NAJA_COLB_DECL)
#undef NAJA_COLB_DECL

int chr_sparse_batch_plan(int m_max, int d, bool quick, BatchConfig* cfg) {
  const int nt = cfg->threads;
  if (nt != 64 && nt != 128 && nt != 256) return NAJA_ERR_INVALID_ARGUMENT;
  if (cfg->slots < 3 || cfg->slots > kMaxSlots) return NAJA_ERR_INVALID_ARGUMENT;
  if (cfg->max_col <= 0) return NAJA_ERR_UNSUPPORTED;
  if (quick && cfg->entries > 0) {
    // A chain's CTA holds the layout, the item's arguments and 1 KB of the
    // system's.  A ring shallower than asked for is taken where it lets one
    // more chain per SM run (a second wave of chains costs as much as the
    // first).
    const size_t fixed = align_up(sizeof(ChrArgs) + sizeof(SpArgs), 128) + 1024;
    auto bytes = [&](int slots) { return make_col_layout(d, m_max, 4, nt / 32, cfg->entries, slots).total; };
    const int most = nt >= 256 ? 2 : (nt == 128 ? 4 : 6);  // chains per SM the registers allow
    auto chains = [&](int slots) {
      const int n = static_cast<int>((kSmemBudget + 1024) / (bytes(slots) + fixed));
      return n < most ? n : most;
    };
    int slots = cfg->slots;
    for (int q = cfg->slots - 1; q >= 3; --q)
      if (chains(q) > chains(slots)) slots = q;
    if (chains(slots) > 0) {
      cfg->slots = slots;
      cfg->rows = 0;
      cfg->lda_max = m_max;
      cfg->smem = bytes(slots);
      return NAJA_OK;
    }
  }
  cfg->entries = 0;
  const Layout L = make_sparse_layout(d, m_max, 4, kSpEntryBytes32, cfg->max_col, nt / 32, cfg->slots);
  // the kernel also holds one ChrArgs and one SpArgs in static shared memory
  if (L.total + align_up(sizeof(ChrArgs) + sizeof(SpArgs), 128) > kSmemBudget) return NAJA_ERR_UNSUPPORTED;
  cfg->rows = 0;
  cfg->lda_max = m_max;
  cfg->smem = L.total;
  return NAJA_OK;
}

int chr_sparse_batch_dispatch(const ChrArgs* base, const ModelDesc* models, const int* im, const int* ic, int nitems,
                              const BatchConfig& cfg, cudaStream_t stream, int* occ_out) {
  if (cfg.entries) {
#define NAJA_COLB_CASE(NW) \
  case 32 * NW: return chr_columns_batch_##NW(base, models, im, ic, nitems, cfg, stream, occ_out);
    switch (cfg.threads) {
      NAJA_COLB_EACH(NAJA_COLB_CASE)
      default: return NAJA_ERR_UNSUPPORTED;
    }
#undef NAJA_COLB_CASE
  }
  switch (cfg.threads) {
    case 64: return batch_sparse_one<2>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 128: return batch_sparse_one<4>(base, models, im, ic, nitems, cfg, stream, occ_out);
    case 256: return batch_sparse_one<8>(base, models, im, ic, nitems, cfg, stream, occ_out);
    default: return NAJA_ERR_UNSUPPORTED;
  }
}
}  // namespace naja
