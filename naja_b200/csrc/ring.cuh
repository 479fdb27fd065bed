// The column ring of the step kernels' producer warps: which slot a step's
// columns take and which phase of the slot's barriers they belong to.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define NAJA_RING_FN __host__ __device__ __forceinline__
#else
#define NAJA_RING_FN inline
#endif

namespace naja {

// Claim p of a launch takes slot p % S in round p / S.  A launch may make any
// number of claims (a chain's steps are counted in 64 bits), and only the
// parity of a round and whether it is the first one matter, so the next claim
// is kept modulo two rounds.
struct RingClaims {
  uint32_t S;              // slots
  uint32_t next = 0;       // the next claim, modulo 2 S
  bool lapped = false;     // every slot has been claimed before
  NAJA_RING_FN explicit RingClaims(int slots) : S(static_cast<uint32_t>(slots)) {}
  // Slot of the claim k after the next one.
  NAJA_RING_FN int slot(uint32_t k) const { return static_cast<int>((next + k) % S); }
  // That claim refills a slot: the slot's release has to be waited for first.
  NAJA_RING_FN bool refill(uint32_t k) const { return lapped || next + k >= S; }
  // Parity of the claim's round: the fill's phase of the slot's full barrier;
  // the release it waits for is the other parity of the empty one.
  NAJA_RING_FN uint32_t parity(uint32_t k) const { return ((next + k) / S) & 1u; }
  NAJA_RING_FN void advance(uint32_t n) {
    lapped = refill(n);
    next = (next + n) % (2 * S);
  }
  // Slot q has been claimed, and the parity of its last fill.
  NAJA_RING_FN bool used(uint32_t q) const { return lapped || q < next; }
  NAJA_RING_FN uint32_t last_parity(uint32_t q) const { return ((next + 2 * S - 1 - q) / S) & 1u; }
};

}  // namespace naja
