// Conversions between FP64, FP32 and double-float pairs in integers, bit for bit
// what the casts give.  A conversion instruction costs the FP64 pipe as much as an
// FMA (16 cycles a warp and SM), rebuilding the exponent about a tenth of it.
// Values that the integer steps do not cover go out of line: predicated in place
// the conversion would take the pipe for every value.  Host and device.
#pragma once

#include <stdint.h>
#include <string.h>

#include "dfloat.cuh"

namespace scft {

#define CV_HD __host__ __device__ __forceinline__
#define CV_RARE __host__ __device__ __noinline__

CV_HD uint32_t float_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u; memcpy(&u, &x, 4); return u;
#endif
}
CV_HD float bits_float(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x; memcpy(&x, &u, 4); return x;
#endif
}
CV_HD uint32_t high_word(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2hiint(x);
#else
  uint64_t u; memcpy(&u, &x, 8); return (uint32_t)(u >> 32);
#endif
}
CV_HD uint32_t low_word(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2loint(x);
#else
  uint64_t u; memcpy(&u, &x, 8); return (uint32_t)u;
#endif
}
CV_HD double words_double(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t u = (uint64_t)hi << 32 | lo;
  double x; memcpy(&x, &u, 8); return x;
#endif
}

// x in FP64
static CV_RARE double widen_rare(float x) { return (double)x; }
CV_HD double widen(double x) { return x; }
CV_HD double widen(float x) {
  const uint32_t u = float_bits(x), m = u & 0x7fffffffu;
  if (m - 0x00800000u >= 0x7f000000u && m != 0u) return widen_rare(x);   // denormal, inf, nan
  const uint32_t hi = (u & 0x80000000u) | (m ? (m >> 3) + 0x38000000u : 0u);
  return words_double(hi, u << 29);
}
CV_HD double widen(dfloat x) { return widen(x.hi) + widen(x.lo); }

// x rounded to the working precision, to nearest even
static CV_RARE float narrow_rare(double x) { return (float)x; }
CV_HD void narrow(double x, double &r) { r = x; }
CV_HD void narrow(double x, dfloat &r) { r = dfloat(x); }
CV_HD void narrow(double x, float &r) {
  const uint32_t hi = high_word(x), lo = low_word(x), m = hi & 0x7fffffffu;
  if (m - 0x38100000u >= 0x0fd00000u && (m | lo) != 0u) {   // below 2^-126, near the top, inf, nan
    r = narrow_rare(x);
    return;
  }
  // 23 bits and the rest below them; a carry moves into the exponent as it should
  const uint32_t f = m ? ((m - 0x38000000u) << 3) | (lo >> 29) : 0u, rest = lo & 0x1fffffffu;
  const uint32_t up = rest > 0x10000000u || (rest == 0x10000000u && (f & 1u)) ? 1u : 0u;
  r = bits_float((hi & 0x80000000u) | (f + up));
}

// dfloat(x); zero, values outside 2^-60 .. 2^120, infinities and NaN out of line
static CV_RARE dfloat pair_rare(double x) { return dfloat(x); }
CV_HD dfloat pair_of(double x) {
  const uint32_t hi = high_word(x), lo = low_word(x), m = hi & 0x7fffffffu;
  if (m - ((1023u - 60u) << 20) >= 180u << 20) return pair_rare(x);
  const uint32_t f = ((m - 0x38000000u) << 3) | (lo >> 29), rest = lo & 0x1fffffffu;
  const uint32_t up = rest > 0x10000000u || (rest == 0x10000000u && (f & 1u)) ? 1u : 0u;
  int r = (int)rest - (int)(up << 29);           // x - hi, in units of 2^(e - 52)
  r = (int)hi < 0 ? -r : r;
  dfloat d;
  d.hi = bits_float((hi & 0x80000000u) | (f + up));
  d.lo = (float)r * bits_float(((m >> 20) - (1023u - 127u) - 52u) << 23);
  return d;
}

#undef CV_HD
#undef CV_RARE

}  // namespace scft
