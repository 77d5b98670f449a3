// Conversions between doubles and floats by integer instructions, host and device,
// the same bits as the casts.
//
// A cast occupies GB300's FP64 pipe like any FP64 instruction, 64 cycles per warp
// and scheduler; these take 5 to 15 integer ones. Only what the fast paths leave
// out (subnormal, infinite, NaN and, for the pair, very large or small values)
// takes the casts.
#pragma once
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define UMCP_CONVERT __host__ __device__ __forceinline__
#else
#define UMCP_CONVERT inline
#endif

namespace umcp {
namespace convert {

UMCP_CONVERT uint64_t bits(double x) {
  uint64_t u;
  memcpy(&u, &x, sizeof u);
  return u;
}
UMCP_CONVERT uint32_t bits(float x) {
  uint32_t u;
  memcpy(&u, &x, sizeof u);
  return u;
}
UMCP_CONVERT float f32_of_bits(uint32_t u) {
  float x;
  memcpy(&x, &u, sizeof x);
  return x;
}

constexpr uint32_t kBiasGap = 1023 - 127;
UMCP_CONVERT uint32_t exponent(uint64_t u) { return (uint32_t)(u >> 52) & 0x7FFu; }
// The 52-bit fraction cut to 23 bits, to nearest even, with the exponent field above it
// (rounding up may carry into it): bits 29 and up of the sum.
UMCP_CONVERT uint32_t rounded(uint64_t u) { return (uint32_t)((u + 0x0FFFFFFFull + ((u >> 29) & 1ull)) >> 29); }
// A float from those bits, its exponent in the normal range, and the sign of u.
UMCP_CONVERT float f32_of_rounded(uint32_t m, uint64_t u) {
  return f32_of_bits(((m - (kBiasGap << 23)) & 0x7FFFFFFFu) | ((uint32_t)(u >> 32) & 0x80000000u));
}

// (float)x
UMCP_CONVERT float to_f32(double x) {
  const uint64_t u = bits(x);
  if (exponent(u) - (kBiasGap + 1) < 253u) return f32_of_rounded(rounded(u), u);
  if ((u << 1) == 0) return f32_of_bits((uint32_t)(u >> 32));
  return (float)x;
}

// (double)x
UMCP_CONVERT double to_f64(float x) {
  const uint32_t b = bits(x);
  if (((b >> 23) & 0xFFu) - 1u >= 254u && (b << 1) != 0) return (double)x;  // subnormal, infinite, NaN
  const uint32_t gap = (b << 1) == 0 ? 0u : kBiasGap << 20;
  const uint64_t u = (uint64_t)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + gap)) << 32 | (uint64_t)(b << 29);
  double y;
  memcpy(&y, &u, sizeof y);
  return y;
}

// hi = (float)x, lo = (float)(x - (double)hi)
UMCP_CONVERT void to_f32_pair(double x, float &hi, float &lo) {
  const uint64_t u = bits(x);
  const uint32_t e = exponent(u);
  if (e - (1023u - 64u) < 128u) {
    const uint32_t m = rounded(u);
    hi = f32_of_rounded(m, u);
    // what was cut off, in units of the last bit of x: the low 29 bits, less 2^29 where
    // the cut rounded up
    const int32_t rest = (int32_t)((uint32_t)u & 0x1FFFFFFFu) - (int32_t)((m - (uint32_t)(u >> 29)) << 29);
    const float unit = f32_of_bits(((e - 52u - kBiasGap) << 23) | ((uint32_t)(u >> 32) & 0x80000000u));
    lo = (float)rest * unit + 0.f;  // + 0: no negative zero
  } else if ((u << 1) == 0) {
    hi = f32_of_bits((uint32_t)(u >> 32));
    lo = 0.f;
  } else {
    hi = (float)x;
    lo = (float)(x - (double)hi);
  }
}

}  // namespace convert
}  // namespace umcp
