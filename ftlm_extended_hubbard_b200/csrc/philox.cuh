// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) and the complex Gaussian start entries drawn from it.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ftlm_b200 {

// 10 rounds of the 4x32 S-box with the published multipliers and Weyl key increments.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(M0, c.x), lo0 = M0 * c.x;
    const uint32_t hi1 = __umulhi(M1, c.z), lo1 = M1 * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += W0;
    k.y += W1;
  }
  return c;
}

// Standard complex Gaussian of state i for a chain's key: counter = i, Box-Muller on two 53-bit uniforms in (0, 1).
__device__ __forceinline__ double2 philox_normal(int64_t i, unsigned key) {
  const uint4 r = philox4x32_10(make_uint4(static_cast<uint32_t>(i), static_cast<uint32_t>(i >> 32), 0u, 0u),
                                make_uint2(key, 0x7F4A7C15u));
  const uint64_t a = (static_cast<uint64_t>(r.x) << 21) ^ (r.y >> 11);
  const uint64_t b = (static_cast<uint64_t>(r.z) << 21) ^ (r.w >> 11);
  const double u1 = (static_cast<double>(a & ((1ull << 53) - 1)) + 0.5) * 0x1.0p-53;
  const double u2 = (static_cast<double>(b & ((1ull << 53) - 1)) + 0.5) * 0x1.0p-53;
  const double rad = sqrt(-2.0 * log(u1));
  double s, c;
  sincospi(2.0 * u2, &s, &c);
  return make_double2(rad * c, rad * s);
}

}  // namespace ftlm_b200
