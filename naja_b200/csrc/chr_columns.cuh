// Compressed-column CHR step kernel with private rows: the single-model and
// batched kernels for constraint matrices whose columns are mostly zero.
//
// Same steps, same arithmetic and the same results, bit for bit, as
// chr_sparse.cuh (which stays for shapes this kernel does not hold): a step
// touches only the rows where its column(s) of A are nonzero.  What bounds it
// is one step's chain of latencies, so that chain is short:
//   * Rows are private to a warp (NW ranges of rows with equally many
//     nonzeros), and a column is stored as the warps read it: E entries
//     (value, row) for each of their lanes, (0, m) where a lane has none, so
//     an entry is one load at a fixed place.  A slack value is read, updated
//     and read again by one warp only: a step needs no barrier for it, and a
//     pair step merges its two columns inside each warp.
//   * A lane's entries of a step are in registers before the step begins.
//   * FP32 quotients without a branch (screen_quotients), extremes as integer
//     keys, one barrier per step; a state warp awaits columns, moves x and
//     saves samples, a producer warp draws 16 steps at a time.
//   * A whose columns fit beside the rest (RES) stays in shared
//     memory: no column is copied or awaited.
// Rows the step does not touch have quotient 0: they cannot be an extreme of
// a step with a positive and a negative quotient.  A step that is not certain
// (as in chr_screen.cuh) divides its entries exactly, and if one end is still
// missing, all rows of the dense A.
#pragma once
#include "chr_screen.cuh"
#include "chr_sparse.cuh"

namespace naja {
namespace chr_detail {
namespace {

constexpr int kColBatch = 16;          // steps drawn together
constexpr int kColRecs = 2 * kColBatch;

struct ColLayout {
  size_t x_off, slot_off, slot_bytes, rec_off, full_off, empty_off, drawn_off, done_off, post_off, red_off, flag_off,
      alpha_off, slack_off, idx_off, total;
  int slots;     // 0: every column is resident at slot_off
};

// Columns of 32 nw e entries; slots = 0: all d of them are kept in shared
// memory.
__host__ __device__ inline ColLayout make_col_layout(int d, int m, int elt, int nw, int e, int slots) {
  const int eb = elt == 4 ? kSpEntryBytes32 : kSpEntryBytes64;
  ColLayout L;
  size_t off = align_up(static_cast<size_t>(d) * 8, 128);
  L.x_off = 0;
  L.slot_off = off;
  L.slot_bytes = static_cast<size_t>(32 * nw * e) * eb;
  L.slots = slots;
  off += L.slot_bytes * (slots ? slots : d);
  L.rec_off = off;
  off += sizeof(StepRec) * kColRecs;
  L.full_off = off;
  off += 8 * static_cast<size_t>(slots);
  L.empty_off = off;
  off += 8 * static_cast<size_t>(slots);
  L.drawn_off = off;
  off += 16;
  L.done_off = off;
  off = align_up(off + 16, 16);
  L.post_off = off;
  off += 16 * 2 * static_cast<size_t>(nw + 1);
  L.red_off = off;
  off += sizeof(RedEntry) * nw;
  L.flag_off = off;
  off += 16;
  L.alpha_off = off;
  off = align_up(off + 16, 16);
  L.slack_off = off;
  off = align_up(off + static_cast<size_t>(m + 1) * elt, 16);
  L.idx_off = off;  // pair steps: where column j holds this row
  off = align_up(off + static_cast<size_t>(m + 1) * (e <= 6 ? 1 : 2), 16);
  L.total = align_up(off, 128);
  return L;
}

// Keys of a warp or block: FP32 the 32-bit keys of ScreenRows<float>, FP64
// the quotients' bits (signed maximum: the largest, unsigned: the most
// negative one).
template <class Real>
struct ColKeys;
template <>
struct ColKeys<float> {
  uint32_t pos, neg;
  __device__ __forceinline__ static ColKeys none() { return ColKeys{0x80000000u, 0u}; }
  __device__ __forceinline__ static ColKeys nan() { return ColKeys{0x7fffffffu, 0u}; }
  __device__ __forceinline__ void reduce() {
    pos = static_cast<uint32_t>(__reduce_max_sync(0xffffffffu, static_cast<int>(pos)));
    neg = __reduce_max_sync(0xffffffffu, neg);
  }
  __device__ __forceinline__ void post(void* p) const { *static_cast<uint2*>(p) = make_uint2(pos, neg); }
  __device__ __forceinline__ void read(const void* p) {
    const uint2 v = *static_cast<const uint2*>(p);
    pos = v.x;
    neg = v.y;
  }
  __device__ __forceinline__ bool certain() const { return screen_certain32(pos, neg); }
  __device__ __forceinline__ float alpha(float u) const {
    const float lo = -rcp_rn(__uint_as_float(pos)), hi = -rcp_rn(__uint_as_float(neg));
    return __fmaf_rn(u, __fsub_rn(hi, lo), lo);
  }
};
template <>
struct ColKeys<double> {
  unsigned long long pos, neg;
  __device__ __forceinline__ static ColKeys none() { return ColKeys{0x8000000000000000ull, 0ull}; }
  __device__ __forceinline__ static ColKeys nan() { return ColKeys{0x7fffffffffffffffull, 0ull}; }
  __device__ __forceinline__ static uint32_t hi(unsigned long long v) { return static_cast<uint32_t>(v >> 32); }
  __device__ __forceinline__ void reduce() {
    const uint32_t ph = static_cast<uint32_t>(__reduce_max_sync(0xffffffffu, static_cast<int>(hi(pos))));
    const uint32_t nh = __reduce_max_sync(0xffffffffu, hi(neg));
    const uint32_t pl = __reduce_max_sync(0xffffffffu, hi(pos) == ph ? static_cast<uint32_t>(pos) : 0u);
    const uint32_t nl = __reduce_max_sync(0xffffffffu, hi(neg) == nh ? static_cast<uint32_t>(neg) : 0u);
    pos = (static_cast<unsigned long long>(ph) << 32) | pl;
    neg = (static_cast<unsigned long long>(nh) << 32) | nl;
  }
  __device__ __forceinline__ void post(void* p) const { *static_cast<ulonglong2*>(p) = make_ulonglong2(pos, neg); }
  __device__ __forceinline__ void read(const void* p) {
    const ulonglong2 v = *static_cast<const ulonglong2*>(p);
    pos = v.x;
    neg = v.y;
  }
  __device__ __forceinline__ bool certain() const { return screen_certain64(hi(pos), hi(neg)); }
  __device__ __forceinline__ double alpha(double u) const {
    return Tier<double>::alpha(__longlong_as_double(static_cast<long long>(pos)),
                               __longlong_as_double(static_cast<long long>(neg)), u);
  }
};

// Where things are in a chain's shared memory.
struct ColShared {
  unsigned char* smem;
  const ColLayout& L;
  __device__ __forceinline__ ColShared(unsigned char* s, const ColLayout& l) : smem(s), L(l) {}
  __device__ __forceinline__ double* xs() const { return reinterpret_cast<double*>(smem + L.x_off); }
  __device__ __forceinline__ StepRec* recs() const { return reinterpret_cast<StepRec*>(smem + L.rec_off); }
  __device__ __forceinline__ uint64_t* full() const { return reinterpret_cast<uint64_t*>(smem + L.full_off); }
  __device__ __forceinline__ uint64_t* empty() const { return reinterpret_cast<uint64_t*>(smem + L.empty_off); }
  __device__ __forceinline__ uint64_t* drawn() const { return reinterpret_cast<uint64_t*>(smem + L.drawn_off); }
  __device__ __forceinline__ uint64_t* done() const { return reinterpret_cast<uint64_t*>(smem + L.done_off); }
  template <class Real>
  __device__ __forceinline__ unsigned char* post(int buf, int nw, int w) const {
    return smem + L.post_off + static_cast<size_t>(buf * (nw + 1) + w) * 2 * sizeof(Real);
  }
  __device__ __forceinline__ RedEntry* red() const { return reinterpret_cast<RedEntry*>(smem + L.red_off); }
  __device__ __forceinline__ volatile int* abort_flag() const {
    return reinterpret_cast<volatile int*>(smem + L.flag_off);
  }
  __device__ __forceinline__ volatile int* stop() const {
    return reinterpret_cast<volatile int*>(smem + L.flag_off) + 2;
  }
  __device__ __forceinline__ double* alpha() const { return reinterpret_cast<double*>(smem + L.alpha_off); }
};

// ------------------------------------------------------------------ producer
template <class Real, class Src, bool RES>
__device__ __noinline__ void run_col_producer(const ChrArgs& a, const SpArgs& sp, Src& src, const ColLayout& L,
                                              unsigned char* smem) {
  constexpr bool kLanes = std::is_same<Src, PhiloxSource>::value;
  const ColShared sh(smem, L);
  const unsigned char* cols = static_cast<const unsigned char*>(sp.lanes);
  const uint32_t col_bytes = static_cast<uint32_t>(L.slot_bytes);
  const int lane = threadIdx.x & 31;
  const long long total = launch_steps(a);
  RingClaims ring(RES ? 1 : L.slots);  // (resident columns: not used)
  unsigned long long w_empty = 0;
  const unsigned long long p_start = clock64();
  bool stop = false;
  for (long long t0 = 0; t0 < total && !stop; t0 += kColBatch) {
    const int n = total - t0 < kColBatch ? static_cast<int>(total - t0) : kColBatch;
    const long long batch_id = t0 / kColBatch;
    StepRec* batch = sh.recs() + (t0 & (kColRecs - 1));
    if constexpr (RES) {
      // the batch two before this one, in the same half, has been stepped
      if (batch_id >= 2) {
        const bool ok = wait_free(sh.done() + (batch_id & 1), static_cast<uint32_t>(((batch_id >> 1) - 1) & 1),
                                  a.timeout_ns, sh.abort_flag());
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0 && !*sh.abort_flag()) set_error(a.err, kDevTimeoutEmpty, -1, 0, static_cast<int>(t0));
          *sh.abort_flag() = 1;
          break;
        }
      }
    }
    auto draw = [&](int k) {
      src.begin_step(static_cast<uint64_t>(a.step_offset + a.t_first + t0 + k));
      StepDir o;
      const bool ok = draw_direction(src, a, o, nullptr, nullptr);
      StepRec& r = batch[k];
      r.kind = o.kind;
      r.ei = o.ei;
      r.ej = o.ej;
      r.flag = !ok ? kRecBad : (fabs(o.ci) <= 4.0 && fabs(o.cj) <= 4.0) ? 0 : kRecWide;
      r.cif = static_cast<float>(o.ci);
      r.cjf = static_cast<float>(o.cj);
      r.uf = static_cast<float>(o.u);
      r.ci = o.ci;
      r.cj = o.cj;
      r.u = o.u;
      return ok;
    };
    if constexpr (kLanes) {
      if (lane < n) draw(lane);
    } else {
      if (lane == 0)
        for (int k = 0; k < n; ++k)
          if (!draw(k)) break;
    }
    __syncwarp();
    int kind = kCoord, ei = 0, ej = 0, bad = 0;
    if (lane < n) {
      const StepRec& r = batch[lane];
      kind = r.kind;
      ei = r.ei;
      ej = r.ej;
      bad = r.flag & kRecBad;
    }
    const uint32_t bads = __ballot_sync(0xffffffffu, bad != 0);
    if constexpr (RES) {
      if (bads) {
        if (lane == __ffs(bads) - 1) set_error(a.err, kDevBadPair, ei, ej, static_cast<int>(t0 + lane));
        *sh.abort_flag() = 1;
        break;  // the batch is not handed over: the state warp gives up its bounded wait
      }
    }
    if (lane == 0) mbar_arrive(sh.drawn() + (batch_id & 1));
    if constexpr (!RES) {
      const uint32_t pairs = __ballot_sync(0xffffffffu, kind == kPair);
      // this lane's first claim, counted from the batch's first
      const uint32_t claim = lane + __popc(pairs & ((1u << lane) - 1u));
      const int sa = ring.slot(claim), sb = ring.slot(claim + 1);
      const uint32_t pa = ring.parity(claim), pb = ring.parity(claim + 1);
      uint32_t claimed = 0;
      for (int k = 0; k < n; ++k) {
        bool ok = true;
        if (lane == k) {
          if (bad) {
            set_error(a.err, kDevBadPair, ei, ej, static_cast<int>(t0 + k));
            ok = false;
          }
          const unsigned long long w0 = a.wait_cycles ? clock64() : 0ull;
          if (ok && ring.refill(claim) && !wait_free(&sh.empty()[sa], pa ^ 1u, a.timeout_ns, sh.abort_flag())) {
            if (!*sh.abort_flag())
              set_error(a.err, kDevTimeoutEmpty, sa, static_cast<int>(pa), static_cast<int>(t0 + k));
            ok = false;
          }
          if (ok && kind == kPair && ring.refill(claim + 1) &&
              !wait_free(&sh.empty()[sb], pb ^ 1u, a.timeout_ns, sh.abort_flag())) {
            if (!*sh.abort_flag())
              set_error(a.err, kDevTimeoutEmpty, sb, static_cast<int>(pb), static_cast<int>(t0 + k));
            ok = false;
          }
          if (a.wait_cycles) w_empty += clock64() - w0;
          if (ok) {
            mbar_arrive_expect_tx(&sh.full()[sa], col_bytes);
            bulk_g2s(smem + L.slot_off + sa * L.slot_bytes, cols + ei * L.slot_bytes, col_bytes, &sh.full()[sa]);
            if (kind == kPair) {
              mbar_arrive_expect_tx(&sh.full()[sb], col_bytes);
              bulk_g2s(smem + L.slot_off + sb * L.slot_bytes, cols + ej * L.slot_bytes, col_bytes, &sh.full()[sb]);
            }
          } else {
            *sh.abort_flag() = 1;
          }
        }
        if (__ballot_sync(0xffffffffu, ok) != 0xffffffffu) {
          stop = true;
          break;
        }
        claimed += 1u + ((pairs >> k) & 1u);
      }
      ring.advance(claimed);
    }
  }
  if (a.wait_cycles) {
    for (int o = 16; o > 0; o >>= 1) w_empty += __shfl_xor_sync(0xffffffffu, w_empty, o);
    if (lane == 0) {
      a.wait_cycles[4 * blockIdx.x + 1] = w_empty;
      a.wait_cycles[4 * blockIdx.x + 3] = clock64() - p_start;
    }
  }
  if constexpr (!RES) {
    // drain: no bulk copy may outlive the CTA
    if (lane < L.slots && ring.used(lane)) {
      const uint32_t last = ring.last_parity(lane);
      if (!mbar_wait_bounded(&sh.full()[lane], last, a.timeout_ns))
        set_error(a.err, kDevTimeoutDrain, lane, static_cast<int>(last), static_cast<int>(ring.next));
    }
    __syncwarp();
  }
}

// MRG32k3a runs come with seeded states (a.rng_state).
template <class Real, bool RES>
__device__ __noinline__ void col_producer_entry(const ChrArgs& a, const SpArgs& sp, const ColLayout& L,
                                                unsigned char* smem, int chain_local) {
  if (a.rng == 0) {
    PhiloxSource src;
    src.k0 = static_cast<uint32_t>(a.seed);
    src.k1 = static_cast<uint32_t>(a.seed >> 32);
    src.chain = static_cast<uint32_t>(a.chain_base + chain_local);
    run_col_producer<Real, PhiloxSource, RES>(a, sp, src, L, smem);
  } else {
    MrgSource src;
    curandStateMRG32k3a* states = reinterpret_cast<curandStateMRG32k3a*>(a.rng_state);
    if ((threadIdx.x & 31) == 0) src.st = states[chain_local];
    run_col_producer<Real, MrgSource, RES>(a, sp, src, L, smem);
    if ((threadIdx.x & 31) == 0) states[chain_local] = src.st;
  }
}

// The state warp's part of a step: x, and the samples saved from it.
template <class Real>
struct ColMover {
  const ChrArgs& a;
  double* xs;
  const Real* alpha;  // [2]
  int chain_local, lane, thin_ctr;
  size_t out_row;
  ScreenStep<Real> step;
  __device__ __forceinline__ ColMover(const ChrArgs& a_, double* xs_, const Real* alpha_, int chain_local_, int lane_)
      : a(a_), xs(xs_), alpha(alpha_), chain_local(chain_local_), lane(lane_) {
    thin_ctr = static_cast<int>(a.t_first % a.thinning);
    out_row = static_cast<size_t>(a.chain_base + chain_local) +
              static_cast<size_t>((a.t_first + a.thinning - 1) / a.thinning) * a.out_nchains;
  }
  __device__ __forceinline__ void read(const StepRec& r) { step.read(r); }
  // Moves x by step t (the record read last), whose alpha is there.
  __device__ __forceinline__ void move(long long t) {
    if (lane == 0) {
      const double a64 = static_cast<double>(*reinterpret_cast<const volatile Real*>(alpha + (t & 1)));
      if (step.kind == kCoord) {
        xs[step.ei] = __dadd_rn(xs[step.ei], a64);
      } else {
        xs[step.ei] = __fma_rn(a64, static_cast<double>(step.ci), xs[step.ei]);
        xs[step.ej] = __fma_rn(a64, static_cast<double>(step.cj), xs[step.ej]);
      }
    }
    if (thin_ctr == 0) {
      __syncwarp();
      const int d = a.d;
      if (a.samples) {
        if (a.out_f64) {
          double* out = reinterpret_cast<double*>(a.samples) + out_row * d;
          for (int j = lane; j < d; j += 32) out[j] = xs[j];
        } else {
          float* out = reinterpret_cast<float*>(a.samples) + out_row * d;
          for (int j = lane; j < d; j += 32) out[j] = __double2float_rn(xs[j]);
        }
      }
      out_row += static_cast<size_t>(a.out_nchains);
      __syncwarp();
    }
    if (++thin_ctr == a.thinning) thin_ctr = 0;
  }
  __device__ __forceinline__ void finish() {
    __syncwarp();
    if (a.X_final)
      for (int j = lane; j < a.d; j += 32) a.X_final[static_cast<size_t>(chain_local) * a.ldx + j] = xs[j];
  }
};

// Barriers over the NW row warps:
//   kBarPost   every row warp has posted the step's extremes; with the state
//              warp, which arrives once the next column to load (EARLY: of the
//              step after the next one) has landed, and takes up the previous
//              step's alpha after it;
//   kBarExact  only inside a step that is not certain;
//   kBarX      with the state warp, around a recompute (this step's alpha is
//              there; x has moved; the slack is new) and after the last step.
//
// ----------------------------------------------------------------- state warp
template <class Real, int NW, bool RES, bool EARLY>
__device__ __forceinline__ void run_col_state(const ChrArgs& a, const ColLayout& L, unsigned char* smem,
                                              int chain_local) {
  constexpr int NB = 32 * NW + 32;
  const ColShared sh(smem, L);
  const int lane = threadIdx.x & 31;
  const int S = L.slots;
  double* xs = sh.xs();
  const long long total = launch_steps(a);
  int slot = 0;
  uint32_t parity = 0;
  unsigned long long w_full = 0;
  const unsigned long long c_start = clock64();
  auto arrived = [&](long long u) -> bool {
    bool ok = true;
    if ((u & (kColBatch - 1)) == 0) {
      const long long batch = u / kColBatch;
      ok = mbar_wait_bounded(sh.drawn() + (batch & 1), static_cast<uint32_t>((batch >> 1) & 1), a.timeout_ns);
    }
    if constexpr (!RES) {
      const unsigned long long w0 = a.wait_cycles ? clock64() : 0ull;
      const int n = ok && sh.recs()[u & (kColRecs - 1)].kind == kPair ? 2 : 1;
      for (int k = 0; k < n && ok; ++k) {
        ok = mbar_wait_bounded(&sh.full()[slot], parity, a.timeout_ns);
        if (++slot == S) {
          slot = 0;
          parity ^= 1u;
        }
      }
      if (a.wait_cycles) w_full += clock64() - w0;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) set_error(a.err, kDevTimeoutFull, slot, static_cast<int>(parity), static_cast<int>(u));
    return ok;
  };
  ColMover<Real> mover(a, xs, reinterpret_cast<const Real*>(sh.alpha()), chain_local, lane);
  int resync_ctr = a.resync > 0 ? static_cast<int>((a.t_first + 1) % a.resync) : 0;
  bool ok = arrived(0);
  if (lane == 0) {
    sh.stop()[0] = ok ? -1 : 0;
    sh.stop()[1] = 0;
    for (int q = 0; q < 2; ++q) ColKeys<Real>::none().post(sh.post<Real>(q, NW, NW));
  }
  named_bar_sync(kBarPost, NB);  // step 0 can be read
  if (EARLY && ok) {
    if (total > 1) ok = arrived(1);
    if (!ok && lane == 0) sh.stop()[1] = 1;
    named_bar_sync(kBarPost, NB);  // step 1 can be read
  }
  bool pending = false;  // step t - 1 has not moved x yet
  for (long long t = 0; t < total && ok; ++t) {
    constexpr int kAhead = EARLY ? 2 : 1;
    if (t + kAhead < total) ok = arrived(t + kAhead);
    if (!ok && lane == 0) {
      // the row warps find the step uncertain and then the flag
      sh.stop()[0] = static_cast<int>(t & 0x7fffffff);
      ColKeys<Real>::nan().post(sh.post<Real>(static_cast<int>(t & 1), NW, NW));
    }
    named_bar_sync(kBarPost, NB);
    if (!ok) break;
    if (pending) mover.move(t - 1);
    mover.read(sh.recs()[t & (kColRecs - 1)]);
    // (a half of the records is free once its last one has been read)
    if (RES && (t & (kColBatch - 1)) == kColBatch - 1) {
      __syncwarp();
      if (lane == 0) mbar_arrive(sh.done() + ((t / kColBatch) & 1));
    }
    pending = true;
    if (a.resync > 0 && t + 1 < total) {
      if (resync_ctr == 0) {
        named_bar_sync(kBarX, NB);
        mover.move(t);
        pending = false;
        named_bar_sync(kBarX, NB);
        named_bar_sync(kBarX, NB);
      }
      if (++resync_ctr == a.resync) resync_ctr = 0;
    }
  }
  if (!ok) {
    *sh.abort_flag() = 1;
    return;
  }
  named_bar_sync(kBarX, NB);
  if (pending) mover.move(total - 1);
  mover.finish();
  if (a.wait_cycles && lane == 0) {
    a.wait_cycles[4 * chain_local + 0] = w_full;
    a.wait_cycles[4 * chain_local + 2] = clock64() - c_start;
  }
}

// ------------------------------------------------------------------ row warps
// EARLY: the next step's entries are loaded while the extremes travel (twice
// the registers); otherwise after the step, for several chains per SM, which
// hide each other's latencies.
template <class Real, int NW, int E, bool RES, bool EARLY>
__device__ __forceinline__ void run_col_rows(const ChrArgs& a, const SpArgs& sp, const ColLayout& L,
                                             unsigned char* smem, int chain_local) {
  using T = Tier<Real>;
  using Acc = typename T::Acc;
  using Ent = SpEntry<Real>;
  using R64 = SpEntry<double>;
  constexpr int NT = 32 * NW, NB = NT + 32;
  const ColShared sh(smem, L);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  Real* slack = reinterpret_cast<Real*>(smem + L.slack_off);
  // A row's place (from 1) among its warp's entries of column j of a pair
  // step, 0 for none, kTaken once column i's entry has taken it.
  using Idx = typename std::conditional<(E <= 6), unsigned char, unsigned short>::type;
  constexpr int kTaken = E <= 6 ? 0xff : 0xffff;
  Idx* idx = reinterpret_cast<Idx*>(smem + L.idx_off);
  const int m = a.m, S = L.slots;

  auto recompute = [&]() {
    const R64* rows = static_cast<const R64*>(sp.row_ent);
    const double* xs = sh.xs();
    for (int r = tid; r < m; r += NT) {
      double acc = 0.0;
      const int k1 = sp.row_start[r + 1];
      for (int k = sp.row_start[r]; k < k1; k += kSpRowGroup) {
        R64 e[kSpRowGroup];
#pragma unroll
        for (int u = 0; u < kSpRowGroup; ++u) e[u] = rows[k + u];
#pragma unroll
        for (int u = 0; u < kSpRowGroup; ++u) acc = __fma_rn(e[u].v, xs[e[u].r], acc);
      }
      slack[r] = T::from64(__dsub_rn(a.b[r], acc));
    }
  };
  for (int r = tid; r <= m; r += NT) idx[r] = 0;
  if (a.slack_in) {
    const Real* si = static_cast<const Real*>(a.slack_in) + static_cast<size_t>(chain_local) * m;
    for (int r = tid; r < m; r += NT) slack[r] = si[r];
  } else {
    recompute();
  }
  if (tid == 0) slack[m] = Real(1);  // the row of lanes without an entry: quotient 0
  named_bar_sync(kBarExact, NT);

  // A step's entries of this lane: value and row, (0, m) where there is none.
  // v1 / r1: of the column (a pair step: of column i, merged with column j's
  // value there); v2 / r2: column j's rows that column i does not hold.
  Real v1[E], v2[E], nv1[E], nv2[E];
  int r1[E], r2[E], nr1[E], nr2[E];
  int slot = 0;
  const int at0 = warp * E * 32 + lane;  // this lane's first entry of a column
  auto column = [&](int j) -> const Ent* {
    const Ent* c = reinterpret_cast<const Ent*>(smem + L.slot_off + (RES ? j : slot) * L.slot_bytes);
    if (!RES && ++slot == S) slot = 0;
    return c;
  };
  // Loads (and merges) a step's entries into nv / nr and gives its slots back.
  auto load = [&](const ScreenStep<Real>& o) {
    const int sa = slot;
    const Ent* ca = column(o.ei);
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const Ent q = ca[at0 + 32 * k];
      nv1[k] = q.v;
      nr1[k] = q.r;
    }
    if (o.kind == kPair) {
      const int sb = slot;
      const Ent* cb = column(o.ej);
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const Ent q = cb[at0 + 32 * k];
        nv2[k] = q.v;
        nr2[k] = q.r;
        if (q.r < m) idx[q.r] = static_cast<Idx>(lane + 32 * k + 1);
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < E; ++k) {
        if (nr1[k] < m) {
          const int at = idx[nr1[k]];
          Real w = Real(0);
          if (at) {
            w = cb[at0 - lane + at - 1].v;
            idx[nr1[k]] = kTaken;
          }
          nv1[k] = T::pair_ae_r(nv1[k], w, o.ci, o.cj);
        }
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < E; ++k) {
        if (nr2[k] < m) {
          const bool taken = idx[nr2[k]] == kTaken;
          idx[nr2[k]] = 0;
          nv2[k] = T::pair_ae_r(Real(0), nv2[k], o.ci, o.cj);
          if (taken) {
            nv2[k] = Real(0);
            nr2[k] = m;
          }
        }
      }
      __syncwarp();
      if (!RES && lane == 0) mbar_arrive(&sh.empty()[sb]);
    } else {
      __syncwarp();
    }
    if (!RES && lane == 0) mbar_arrive(&sh.empty()[sa]);
  };
  auto take = [&]() {
#pragma unroll
    for (int k = 0; k < E; ++k) {
      v1[k] = nv1[k];
      r1[k] = nr1[k];
      v2[k] = nv2[k];
      r2[k] = nr2[k];
    }
  };

  const long long total = launch_steps(a);
  int resync_ctr = a.resync > 0 ? static_cast<int>((a.t_first + 1) % a.resync) : 0;
  ScreenStep<Real> cur, nxt;
  named_bar_sync(kBarPost, NB);  // step 0 has arrived
  if (sh.stop()[0] >= 0) return;
  cur.read(sh.recs()[0]);
  load(cur);
  take();
  if constexpr (EARLY) {
    named_bar_sync(kBarPost, NB);  // step 1 has arrived
    if (sh.stop()[1]) return;
  }
  for (long long t = 0; t < total; ++t) {
    const int buf = static_cast<int>(t & 1);
    const bool more = t + 1 < total;
    if (EARLY) nxt.read(sh.recs()[(t + 1) & (kColRecs - 1)]);
    Real s1[E], s2[E];
#pragma unroll
    for (int k = 0; k < E; ++k) s1[k] = slack[r1[k]];
    const bool pair = cur.kind == kPair;
    if (pair) {
#pragma unroll
      for (int k = 0; k < E; ++k) s2[k] = slack[r2[k]];
    }
    ColKeys<Real> e;
    if constexpr (sizeof(Real) == 4) {
      ScreenAcc acc;
      screen_quotients<E>(v1, s1, acc);
      if (pair) screen_quotients<E>(v2, s2, acc);
      e.pos = acc.pos_key();
      e.neg = acc.neg;
    } else {
      e.pos = 0x8000000000000000ull;
      e.neg = 0ull;
      auto add = [&](double v, double s) {
        const unsigned long long q = static_cast<unsigned long long>(__double_as_longlong(T::ratio(v, s)));
        e.pos = static_cast<long long>(q) > static_cast<long long>(e.pos) ? q : e.pos;
        e.neg = q > e.neg ? q : e.neg;
      };
#pragma unroll
      for (int k = 0; k < E; ++k) add(v1[k], s1[k]);
      if (pair) {
#pragma unroll
        for (int k = 0; k < E; ++k) add(v2[k], s2[k]);
      }
    }
    e.reduce();
    if (lane == 0) e.post(sh.post<Real>(buf, NW, warp));
    // the next step's entries, while the other warps post
    if (EARLY && more) load(nxt);
    named_bar_sync(kBarPost, NB);
    if constexpr (NW > 1) {
      e.read(sh.post<Real>(buf, NW, lane <= NW ? lane : NW));  // the state warp's entry counts only when it gave up
      e.reduce();
    } else {
      if (sh.stop()[0] >= 0) return;
    }
    Real alpha;
    if (e.certain() && cur.flag == 0) {
      alpha = e.alpha(cur.u);
    } else {
      if (sh.stop()[0] == static_cast<int>(t & 0x7fffffff)) return;
      // exactly: this step's entries, then, if an end is missing, all rows
      Acc h, l, l2;
      auto block = [&]() {
        h = T::red_hi(h);
        l = T::red_lo(l);
        l2 = T::red_lo2(l2);
        if constexpr (NW > 1) {
          if (lane == 0) {
            sh.red()[warp].kmax = h;
            sh.red()[warp].kmin = l;
            sh.red()[warp].kmin2 = l2;
          }
          named_bar_sync(kBarExact, NT);
          h = T::acc_hi0();
          l = T::acc_lo0();
          l2 = T::acc_lo20();
          if (lane < NW) {
            h = static_cast<Acc>(sh.red()[lane].kmax);
            l = static_cast<Acc>(sh.red()[lane].kmin);
            l2 = static_cast<Acc>(sh.red()[lane].kmin2);
          }
          named_bar_sync(kBarExact, NT);
          h = T::red_hi(h);
          l = T::red_lo(l);
          l2 = T::red_lo2(l2);
        }
      };
      h = T::acc_hi0();
      l = T::acc_lo0();
      l2 = T::acc_lo20();
#pragma unroll 1
      for (int k = 0; k < (pair ? 2 * E : E); ++k) {
        Real cv = v1[0], cs = s1[0];
        int cr = r1[0];
        const uint32_t bit = 1u << k;  // (a bit: an index would put the arrays in local memory)
#pragma unroll
        for (int i = 0; i < E; ++i) {
          if (bit & (1u << i)) {
            cv = v1[i];
            cs = s1[i];
            cr = r1[i];
          }
          if (bit & (1u << (E + i))) {
            cv = v2[i];
            cs = s2[i];
            cr = r2[i];
          }
        }
        if (cr < m) T::acc(h, l, l2, T::ratio(cv, cs));
      }
      block();
      Real mx, mn;
      T::decode(h, l, l2, mx, mn);
      if (!(mx > Real(0) && mn < Real(0))) {
        h = T::acc_hi0();
        l = T::acc_lo0();
        l2 = T::acc_lo20();
        const Real* ca = T::A(a) + static_cast<size_t>(cur.ei) * a.lda;
        const Real* cb = T::A(a) + static_cast<size_t>(pair ? cur.ej : 0) * a.lda;
        for (int r = tid; r < m; r += NT)
          T::acc(h, l, l2, T::ratio(pair ? T::pair_ae_r(ca[r], cb[r], cur.ci, cur.cj) : ca[r], slack[r]));
        block();
        T::decode(h, l, l2, mx, mn);
      }
      alpha = T::alpha(mx, mn, cur.u);
      // (a dense pass of another warp may still be reading this one's rows)
      if constexpr (NW > 1) named_bar_sync(kBarExact, NT);
    }
    if (tid == 0) reinterpret_cast<volatile Real*>(sh.alpha())[buf] = alpha;
    bool again = false;
    if (a.resync > 0 && more) {
      again = resync_ctr == 0;
      if (++resync_ctr == a.resync) resync_ctr = 0;
    }
    if (again) {
      named_bar_sync(kBarX, NB);
      named_bar_sync(kBarX, NB);  // the state warp has moved x
      recompute();
      named_bar_sync(kBarX, NB);
    } else {
#pragma unroll
      for (int k = 0; k < E; ++k) slack[r1[k]] = T::slack_update(s1[k], alpha, v1[k]);
      if (pair) {
#pragma unroll
        for (int k = 0; k < E; ++k) slack[r2[k]] = T::slack_update(s2[k], alpha, v2[k]);
      }
      __syncwarp();
    }
    if (!EARLY) nxt.read(sh.recs()[(t + 1) & (kColRecs - 1)]);
    if (!EARLY && more) load(nxt);
    take();
    cur = nxt;
  }
  named_bar_sync(kBarX, NB);
  if (a.slack_final) {
    named_bar_sync(kBarExact, NT);
    Real* so = static_cast<Real*>(a.slack_final) + static_cast<size_t>(chain_local) * m;
    for (int r = tid; r < m; r += NT) so[r] = slack[r];
  }
}

// Everything of one chain before its steps: barriers, x, resident columns.
template <class Real, int NW, bool RES>
__device__ __forceinline__ void col_prologue(const ChrArgs& a, const SpArgs& sp, const ColLayout& L,
                                             unsigned char* smem, int chain_local) {
  const ColShared sh(smem, L);
  if (threadIdx.x == 0) {
    for (int q = 0; q < L.slots; ++q) {
      mbar_init(&sh.full()[q], 1);
      mbar_init(&sh.empty()[q], NW);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(sh.drawn() + q, 1);
      mbar_init(sh.done() + q, 1);
    }
    fence_mbar_init();
  }
  for (int j = threadIdx.x; j < a.d; j += 32 * NW + 64)
    sh.xs()[j] = a.X0[static_cast<size_t>(chain_local) * a.ldx + j];
  if constexpr (RES) {
    const uint4* src = static_cast<const uint4*>(sp.lanes);
    const size_t n16 = a.d * L.slot_bytes / 16;
    for (size_t i = threadIdx.x; i < n16; i += 32 * NW + 64) reinterpret_cast<uint4*>(smem + L.slot_off)[i] = src[i];
  }
}

template <class Real, int NW, int E, bool RES>
__global__ void __launch_bounds__(NW * 32 + 64, 1)
    chr_columns_kernel(const __grid_constant__ ChrArgs a, const __grid_constant__ SpArgs sp,
                       const __grid_constant__ ColLayout L) {
  extern __shared__ __align__(128) unsigned char smem[];
  if (threadIdx.x == 0) *ColShared(smem, L).abort_flag() = 0;
  col_prologue<Real, NW, RES>(a, sp, L, smem, blockIdx.x);
  __syncthreads();
  if (threadIdx.x >= NW * 32 + 32) {
    col_producer_entry<Real, RES>(a, sp, L, smem, blockIdx.x);
  } else if (threadIdx.x >= NW * 32) {
    run_col_state<Real, NW, RES, true>(a, L, smem, blockIdx.x);
  } else {
    run_col_rows<Real, NW, E, RES, true>(a, sp, L, smem, blockIdx.x);
  }
}

// Batched multi-model run: the persistent item loop of chr_batched_kernel
// (one item = one chain of one model) over the kernel above, columns staged.
// Layout for the largest model, lane order of E entries for every model.
template <int NW, int E>
__global__ void __launch_bounds__(NW * 32 + 64, NW >= 8 ? 2 : (NW == 4 ? 4 : 6))
    chr_batched_columns_kernel(const __grid_constant__ ChrArgs base, const __grid_constant__ ColLayout L,
                               const ModelDesc* __restrict__ models, const int* __restrict__ item_model,
                               const int* __restrict__ item_chain, int nitems) {
  using Real = float;
  constexpr int NT = NW * 32;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ChrArgs item_args;
  __shared__ SpArgs item_sp;
  const ColShared sh(smem, L);
  if (threadIdx.x == 0) *sh.abort_flag() = 0;
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int ch = item_chain[item];
    if (threadIdx.x == 0) {
      item_args = item_arguments(base, models[item_model[item]]);
      item_sp = models[item_model[item]].sp;
    }
    __syncthreads();
    if (*sh.abort_flag()) break;  // every thread reads it after the barrier
    col_prologue<Real, NW, false>(item_args, item_sp, L, smem, ch);
    __syncthreads();
    if (threadIdx.x >= NT + 32) {
      col_producer_entry<Real, false>(item_args, item_sp, L, smem, ch);
    } else if (threadIdx.x >= NT) {
      run_col_state<Real, NW, false, false>(item_args, L, smem, ch);
    } else {
      run_col_rows<Real, NW, E, false, false>(item_args, item_sp, L, smem, ch);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int q = 0; q < L.slots; ++q) {
        mbar_inval(&sh.full()[q]);
        mbar_inval(&sh.empty()[q]);
      }
      for (int q = 0; q < 2; ++q) {
        mbar_inval(sh.drawn() + q);
        mbar_inval(sh.done() + q);
      }
    }
  }
}

template <int NW, int E>
int batch_columns_one(const ChrArgs* base, const ModelDesc* models, const int* im, const int* ic, int nitems,
                      const BatchConfig& cfg, cudaStream_t stream, int* occ_out) {
  return batch_run(chr_batched_columns_kernel<NW, E>, NW * 32 + 64, align_up(sizeof(ChrArgs) + sizeof(SpArgs), 128), cfg,
                   nitems, occ_out, [&](auto kern, int grid) {
    const ColLayout L = make_col_layout(base->d, cfg.lda_max, sizeof(float), NW, E, cfg.slots);
    kern<<<grid, NW * 32 + 64, cfg.smem, stream>>>(*base, L, models, im, ic, nitems);
  });
}

}  // namespace
}  // namespace chr_detail
}  // namespace naja
