// The producers' column ring against 64-bit arithmetic on the claim's number,
// from a launch's first claim and across claim 2^32.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "../../naja_b200/csrc/ring.cuh"

static int bad(const char* what, int S, unsigned long long p) {
  std::printf("%s: %d slots, claim %llu\n", what, S, p);
  return 1;
}

static int walk(int S, unsigned long long first, int batches) {
  naja::RingClaims ring(S);
  // the state after `first` claims
  ring.next = static_cast<uint32_t>(first % (2ull * S));
  ring.lapped = first >= static_cast<unsigned long long>(S);
  unsigned long long p = first;
  std::srand(S);
  for (int b = 0; b < batches; ++b) {
    const uint32_t n = 1 + std::rand() % 64;  // up to 32 steps of one or two columns
    for (uint32_t k = 0; k <= n; ++k) {
      const unsigned long long q = p + k, round = q / S;
      if (ring.slot(k) != static_cast<int>(q % S)) return bad("slot", S, q);
      if (ring.refill(k) != (round >= 1)) return bad("refill", S, q);
      if (ring.parity(k) != (round & 1)) return bad("parity", S, q);
    }
    ring.advance(n);
    p += n;
    for (int q = 0; q < S; ++q) {
      const bool used = p > static_cast<unsigned long long>(q);
      if (ring.used(q) != used) return bad("used", S, p);
      if (used && ring.last_parity(q) != (((p - 1 - q) / S) & 1)) return bad("last", S, p);
    }
  }
  return 0;
}

int main() {
  for (int S = 3; S <= 8; ++S)
    for (unsigned long long first : {0ull, 1ull, (1ull << 32) - 700, (1ull << 33) - 700, (1ull << 62) - 700})
      if (walk(S, first, 100)) return 1;
  std::printf("ring ok\n");
  return 0;
}
