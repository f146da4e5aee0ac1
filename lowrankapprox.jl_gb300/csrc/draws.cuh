// The draws of a Gaussian sketch on the device: the 1/32 lattice and the
// in-library generator.
#pragma once

#include <stdint.h>

namespace lra {

// 32 g rounded to the nearest integer (ties to even) and clipped to +-127, from
// the bits of g: the FP64 unit takes 64 cycles a warp instruction, and rounding
// and clipping there costs eight of them
__device__ __forceinline__ int lattice_int(double g) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(g);
  const int e = (int)(b >> 52) & 0x7ff;
  // 32 |g| = M 2^-s, M the 53-bit mantissa
  const int s = 1070 - e;
  int k;
  if (s >= 55) {
    k = 0;  // below 1/4
  } else if (s <= 45) {
    // 128 and more; a NaN clips to -127, as fmax and fmin take it
    return (b >> 63) || (e == 0x7ff && (b & 0xfffffffffffffull)) ? -127 : 127;
  } else {
    const unsigned long long M = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const unsigned long long rem = M & ((1ull << s) - 1), half = 1ull << (s - 1);
    k = (int)(M >> s);
    k += rem > half || (rem == half && (k & 1)) ? 1 : 0;
    k = k > 127 ? 127 : k;
  }
  return (b >> 63) ? -k : k;
}

// the same rounding in FP32 (exact: the lattice values are k / 32, |k| <= 127)
__device__ __forceinline__ float lattice_f(float g) {
  const float r = fminf(127.0f, fmaxf(-127.0f, rintf(g * 32.0f)));
  return r * 0.03125f;
}

// Philox-4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11), own implementation.
struct U4 {
  unsigned x, y, z, w;
};
__device__ __forceinline__ U4 philox(U4 c, unsigned k0, unsigned k1) {
  const unsigned M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned hi0 = __umulhi(M0, c.x), lo0 = M0 * c.x;
    const unsigned hi1 = __umulhi(M1, c.z), lo1 = M1 * c.z;
    c = U4{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
    k0 += W0;
    k1 += W1;
  }
  return c;
}

// two Gaussians from a counter's output: Box-Muller on two uniforms in (0, 1],
// in FP32: the draws are rounded to the 1/32 lattice, far coarser than FP32's
// resolution, and FP64 transcendentals are slow on this part
__device__ __forceinline__ float2 philox_gauss(U4 r) {
  const float u1 = ((float)r.x + 1.0f) * 2.3283064365386963e-10f;
  const float u2 = ((float)r.y + 0.5f) * 2.3283064365386963e-10f;
  const float rad = sqrtf(-2.0f * logf(u1));
  float s, c;
  sincospif(2.0f * u2, &s, &c);
  return make_float2(rad * c, rad * s);
}

// draw t of the generator at counter `base` (draws 2 q and 2 q + 1 share counter
// base + q)
__device__ __forceinline__ float2 philox_pair(uint64_t seed, uint64_t base, int64_t q) {
  const uint64_t ctr = base + (uint64_t)q;
  return philox_gauss(
      philox(U4{(unsigned)ctr, (unsigned)(ctr >> 32), 0x6c72u, 0x61u}, (unsigned)seed, (unsigned)(seed >> 32)));
}

}  // namespace lra
