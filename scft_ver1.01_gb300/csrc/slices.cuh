// Fixed-point slices for the tensor-core line filter (k_tc.cu): conversions
// between the working reals and line-scaled integers, and the integers' signed
// base-256 digits.  Host and device, integer and FP32 arithmetic only: an FP64
// instruction on GB300 takes 16 cycles of an SM per warp, the sequences here
// 3 to 6.
//
// A line x is held as integers X with x = X * 2^ue, ue chosen from the line's
// largest exponent so that |X| <= 2^54 (FP64; 7 digits) or 2^29
// (FP32; 4 digits).  All roundings are to nearest: a truncation's bias would
// add up over the contour steps.  Denormals are kept.
#pragma once

#include <stdint.h>
#include <string.h>

#include "common.cuh"

namespace scft {
namespace slices {

#define SL_HD __host__ __device__ __forceinline__

SL_HD uint32_t f2u(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u; memcpy(&u, &f, 4); return u;
#endif
}
SL_HD float u2f(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f; memcpy(&f, &u, 4); return f;
#endif
}
SL_HD uint64_t d2u(double d) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(d);
#else
  uint64_t u; memcpy(&u, &d, 8); return u;
#endif
}
SL_HD double u2d(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double d; memcpy(&d, &u, 8); return d;
#endif
}
SL_HD int clz64(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)u);
#else
  return u ? __builtin_clzll(u) : 64;
#endif
}
SL_HD int clz32(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __clz((int)u);
#else
  return u ? __builtin_clz(u) : 32;
#endif
}
// A factor W > 0: W = (h * 2^31 + l) * 2^(e - 1022 - 62), h and l two 31-bit halves of its
// 53 bits, normalised (h >= 2^30).
struct Factor {
  int h, l, e;
};
// e of a factor that is not a finite positive number (or of such a real, below):
// far above any other exponent
constexpr int kBadFactor = 1 << 18;
SL_HD bool factor_rare(uint64_t w) {   // not within 2^-500 .. 2^500
  return (uint32_t)(w >> 32) - ((1023u - 500u) << 20) >= 1000u << 20;
}
SL_HD Factor factor_of(uint64_t w) {   // (a normal number)
  const uint32_t hi = (uint32_t)(w >> 32), lo = (uint32_t)w;
  Factor f;
  f.e = (int)(hi >> 20);
  f.h = (int)(((hi & 0x000fffffu) | 0x00100000u) << 10 | lo >> 22);
  f.l = (int)((lo << 9) & 0x7fffffffu);
  return f;
}
static __host__ __device__ __noinline__ Factor factor_of_rare(uint64_t w) {
  Factor f = {0, 0, 0};
  if (w - 0x0010000000000000ULL < 0x7fe0000000000000ULL) {
    f = factor_of(w);
  } else if (w >= 0x7ff0000000000000ULL) {   // negative, infinite, NaN
    f.e = w == 0x8000000000000000ULL ? 0 : kBadFactor;
  } else if (w != 0) {
    const int lz = clz64(w) - 11;      // denormal: its leading bit to bit 52
    const uint64_t m = w << (lz + 9);
    f.e = 1 - lz;
    f.h = (int)(m >> 31);
    f.l = (int)(m & 0x7fffffff);
  }
  return f;
}
// y * (h * 2^31 + l) / 2^62, |y| < 2^61, rounded to nearest but for the product of the
// low halves, which counts with its mean (half of l: within half a unit).
SL_HD int64_t mul_w62(int64_t y, const Factor &w) {
  const int yh = (int)(y >> 31), yl = (int)((uint32_t)y & 0x7fffffffu);
  const int64_t t = (int64_t)yh * w.l + ((int64_t)yl * w.h + (int64_t)((1u << 30) + ((uint32_t)w.l >> 1)));
  return (int64_t)yh * w.h + (t >> 31);
}
// x = m * 2^u, |m| in [2^60, 2^61) or 0; u of kBadFactor: not finite
SL_HD bool real_rare(uint64_t x) {   // zero, denormal, not finite
  return ((uint32_t)(x >> 32) & 0x7fffffffu) - 0x00100000u >= 0x7fe00000u;
}
SL_HD int64_t split_real(uint64_t x, int &u) {   // (a normal number)
  u = ((int)(x >> 52) & 0x7ff) - 1083;
  const int64_t m = (int64_t)(((x & 0xfffffffffffffULL) | 0x10000000000000ULL) << 8), s = (int64_t)x >> 63;
  return (m ^ s) - s;
}
static __host__ __device__ __noinline__ int64_t split_real_rare(uint64_t x, int &u) {
  const uint64_t a = x & 0x7fffffffffffffffULL;
  const int lz = a ? clz64(a) - 11 : 0;          // denormal: its leading bit to bit 52
  u = a >= 0x7ff0000000000000ULL ? kBadFactor : 1 - lz - 1083;
  const int64_t m = a >= 0x7ff0000000000000ULL ? 0 : (int64_t)(a << (lz + 8));
  return (int64_t)x < 0 ? -m : m;
}
// |x| <= 2^bits_of(x), at least 55
SL_HD int bits_of(int64_t x) {
  const int h = (int)(x >> 32);
  return 64 - clz32((uint32_t)(h ^ (h >> 31)) | 0x400000u);
}
// x * 2^-s rounded to nearest (halves up), s > 0
SL_HD int64_t shifted(int64_t x, int s) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s - 1));   // (63 and more: the sign)
  return (r + 1) >> 1;
#else
  return ((x >> (s > 64 ? 63 : s - 1)) + 1) >> 1;
#endif
}

// 2^e as a float, e clamped to the normal range.
SL_HD float exp2i(int e) {
  e = e < -126 ? -126 : (e > 127 ? 127 : e);
  return u2f((uint32_t)(e + 127) << 23);
}
// x * 2^e for any e (two steps keep the factors normal).
SL_HD float scale2(float x, int e) {
  const int h = e / 2;
  return x * exp2i(h) * exp2i(e - h);
}

// Magnitude keys: ordered like |x|; a key of kBadKey<T> or more marks a NaN or
// an infinity.
SL_HD int mag_key(double x) { return (int)((uint32_t)(d2u(x) >> 32) & 0x7fffffffu); }
SL_HD int mag_key(float x) { return (int)(f2u(x) & 0x7fffffffu); }
template <typename T> SL_HD constexpr int bad_key() { return sizeof(T) == 8 ? 0x7ff00000 : 0x7f800000; }

// Biased exponent of a line's largest magnitude, and the unit exponent ue
// (denormals count as exponent 1, which is their unit).
SL_HD int line_exp(double, int key) { return key < 1 << 21 ? 1 : key >> 20; }
SL_HD int line_exp(float, int key) { return key < 1 << 24 ? 1 : key >> 23; }
SL_HD int unit_exp(double, int E) { return E - 1076; }   // |X| < 2^54
SL_HD int unit_exp(float, int E) { return E - 155; }     // |X| <= 2^29

// x / 2^unit_exp(E), rounded to nearest; E is at least x's own exponent.
SL_HD int64_t to_fixed(double x, int E) {
  const uint64_t b = d2u(x);
  const int e = (int)(b >> 52) & 0x7ff;
  const uint64_t m = ((b & 0xfffffffffffffULL) | (e ? 0x10000000000000ULL : 0)) << 8;   // 61 bits
  int sh = E - (e ? e : 1);
  if (sh > 63) sh = 63;                            // far below the line's unit
  const int64_t t = (int64_t)(((m >> sh) + 64) >> 7);
  const int64_t s = (int64_t)b >> 63;
  return (t ^ s) - s;
}
SL_HD int to_fixed(float x, int E) {
  // (2^154 at most: two factors)
  const float s = x * exp2i(E < 29 ? 126 : 155 - E) * exp2i(E < 29 ? 29 - E : 0);
#ifdef __CUDA_ARCH__
  return __float2int_rn(s);
#else
  return (int)lrintf(s);
#endif
}

// y * 2^ue as an FP64 number, |y| < 2^63, rounded to nearest (halves up).
SL_HD double from_fixed(int64_t y, int ue, double) {
  const int64_t sg = y >> 63;
  const uint64_t u = (uint64_t)((y ^ sg) - sg);
  const int lz = clz64(u);                         // >= 1
  const uint64_t m = ((u << ((lz - 1) & 63)) + 0x200) >> 10;   // leading bit 52 (53 after a carry)
  const int be = 1086 + ue - lz;                   // biased exponent of the leading bit
  uint32_t hi = (uint32_t)(m >> 32) + ((uint32_t)(be - 1) << 20), lo = (uint32_t)m;
  if (u == 0) hi = lo = 0;
  else if (be >= 2047) { hi = 0x7ff00000u; lo = 0; }
  else if (be <= 0) {                              // in units of 2^-1074
    const int s = -1074 - ue;                      // (> 0 for |y| >= 2^52)
    const uint64_t d = s > 63 ? 0 : (s > 0 ? (u + (1ULL << (s - 1))) >> s : u << -s);
    hi = (uint32_t)(d >> 32);
    lo = (uint32_t)d;
  }
  return u2d(((uint64_t)(hi | ((uint32_t)(sg >> 32) & 0x80000000u)) << 32) | lo);
}
// The same for |y| in [2^32, 2^62) and results in the normal range (fast path;
// a negative y is taken as ~y, one unit off).
SL_HD double from_fixed_fast(int64_t y, int ue) {
  const uint32_t sg = (uint32_t)(y >> 63);
  const uint32_t h = (uint32_t)(y >> 32) ^ sg, l = (uint32_t)y ^ sg;
  const int lz = clz32(h);                         // 2 .. 31
  const uint64_t m = ((((uint64_t)h << 32 | l) << (lz - 1)) + 0x200) >> 10;
  const uint32_t hi = (uint32_t)(m >> 32) + ((uint32_t)(1085 + ue - lz) << 20);
  return u2d((uint64_t)(hi | (sg & 0x80000000u)) << 32 | (uint32_t)m);
}
SL_HD bool fast_units(int ue) { return (uint32_t)(ue + 1000) < 1900u; }   // -1000 .. 899
// The signed base-256 digits of X (digit i weighs 256^(ND-1-i)) as bytes plus
// 128: all but the top one are in [0, 255]; the top one, in the high half word,
// is in [0, 256] (7 digits) or [64, 192] (4 digits).
SL_HD uint64_t biased_digits(int64_t X) { return (uint64_t)X + 0x0080808080808080ULL; }
SL_HD uint32_t biased_digits(int X) { return (uint32_t)X + 0x80808080u; }

}  // namespace slices
}  // namespace scft
