// Host check of the integer conversions (convert.cuh) against the casts, bit for
// bit: every float by strides, doubles around every rounding tie, carry and edge
// of the integer steps' range.  Prints the number compared and of mismatches.
#include <math.h>
#include <stdio.h>

#include "convert.cuh"

using namespace scft;

static long long n = 0, bad = 0;
static double of_bits(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
static bool same(float a, float b) { return memcmp(&a, &b, 4) == 0 || (isnan(a) && isnan(b)); }
static bool same(double a, double b) { return memcmp(&a, &b, 8) == 0 || (isnan(a) && isnan(b)); }
static void wide(uint32_t u) {
  const float x = bits_float(u);
  ++n;
  bad += !same(widen(x), (double)x);
}
static void from(uint64_t u) {
  const double x = of_bits(u);
  float r;
  narrow(x, r);
  const dfloat p = pair_of(x), q(x);
  n += 2;
  bad += !same(r, (float)x);
  bad += !same(p.hi, q.hi) || !same(p.lo, q.lo);
}

int main() {
  for (uint64_t u = 0; u < 1ull << 32; u += 241) wide((uint32_t)u);
  for (uint32_t e = 0; e < 512; ++e)
    for (int d = -3; d <= 3; ++d) wide((e << 23) + d);
  uint64_t s = 1;
  for (uint64_t se = 0; se < 4096; ++se) {          // sign and exponent
    const uint64_t b = se << 52;
    for (int d = -3; d <= 3; ++d) {
      from(b + d);
      for (uint64_t f : {0ull, 1ull, 2ull, 0x3ffffeull, 0x3fffffull, 0x7ffffeull, 0x7fffffull})
        for (uint64_t r : {0ull, 0x10000000ull, 0x1fffffffull})   // fraction, and the rest below it
          from(b + (f << 29) + r + d);
    }
    for (int k = 0; k < 2000; ++k) {
      s = s * 6364136223846793005ull + 1442695040888963407ull;
      from(b | s >> 12);
      from(b | (s >> 12 & ~0x1fffffffull) | 0x10000000ull);       // a tie
    }
  }
  printf("%lld %lld\n", n, bad);
  return 0;
}
