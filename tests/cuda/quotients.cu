// Counts of disagreement of the screened kernel's branch-free arithmetic with
// the IEEE operations, over ranges of operands.
#include "../../naja_b200/csrc/chr_screen.cuh"

namespace naja {
namespace chr_detail {

// Every significand at binary exponent e, both signs: reciprocals.
__global__ void reciprocals(int e, unsigned long long* bad) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;  // < 2^24
  const float x = __uint_as_float(((i >> 23) << 31) | (static_cast<uint32_t>(e + 127) << 23) | (i & 0x7fffffu));
  if (__float_as_uint(rcp_rn(x)) != __float_as_uint(__fdiv_rn(1.0f, x))) atomicAdd(bad, 1ull);
}

// Quotients of random operands in the range of a certain step: slack 2^-42 ..
// 2^40, |ae| up to 2^61, |ae / s| at least 2^-60.
__global__ void quotients(uint32_t seed, unsigned long long* bad, unsigned long long* tried) {
  const Philox4 r = philox4x32_10(blockIdx.x, threadIdx.x, 0u, 0u, seed, 1u);
  const float s = __uint_as_float((static_cast<uint32_t>(127 - 42 + r.v[0] % 82u) << 23) | (r.v[1] & 0x7fffffu));
  const float a = __uint_as_float((r.v[2] & 0x80000000u) | (static_cast<uint32_t>(127 - 60 + (r.v[2] >> 8) % 121u) << 23) |
                                  (r.v[3] & 0x7fffffu));
  const float q = __fdiv_rn(a, s);
  if (fabsf(q) < 0x1p-60f) return;
  atomicAdd(tried, 1ull);
  ScreenAcc acc;
  acc.add(f2(s, s), f2(a, a));
  const uint32_t got = a < 0.0f ? static_cast<uint32_t>(acc.pos) : acc.neg;  // the bits of -q
  if ((got ^ 0x80000000u) != __float_as_uint(q)) atomicAdd(bad, 1ull);
}

// Every 20-bit fraction at binary exponent e: relative error of the FP64 key's
// reciprocal, low word zero and all ones.
__global__ void estimates(int e, double* worst0, double* worst1) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;  // < 2^20
  const uint32_t hi = (static_cast<uint32_t>(e + 1023) << 20) | i;
  for (int k = 0; k < 2; ++k) {
    const double x = __hiloint2double(static_cast<int>(hi), k ? -1 : 0);
    const double r = __hiloint2double(static_cast<int>(ScreenRows<double, 32, 1, true>::key(1.0, x)), 0);
    const double err = fabs(__fma_rn(r, x, -1.0));
    atomicMax(reinterpret_cast<unsigned long long*>(k ? worst1 : worst0),
              static_cast<unsigned long long>(__double_as_longlong(err)));
  }
}
}  // namespace chr_detail
}  // namespace naja

using namespace naja::chr_detail;

extern "C" int check_reciprocals(int e, unsigned long long* bad) {
  reciprocals<<<1 << 16, 256>>>(e, bad);
  return cudaDeviceSynchronize();
}
extern "C" int check_quotients(unsigned seed, unsigned long long* bad, unsigned long long* tried) {
  quotients<<<1 << 18, 256>>>(seed, bad, tried);
  return cudaDeviceSynchronize();
}
extern "C" int check_estimates(int e, double* worst0, double* worst1) {
  estimates<<<1 << 12, 256>>>(e, worst0, worst1);
  return cudaDeviceSynchronize();
}
