// Host check of the tensor-core line filter's arithmetic (k_tc.cu,
// slices.cuh): line -> integers -> digits, digit products with the table that
// tc_build_table makes, recombination, against a long double convolution with
// the same gains.  Prints one line per case: kind n max-relative-error and the
// largest accumulator.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "tc_core.cuh"


using namespace scft;
using namespace scft::slices;

static double f16(uint16_t h) {
  const int e = (h >> 10) & 31, m = h & 1023;
  const double v = e ? ldexp(1024 + m, e - 25) : ldexp(m, -24);
  return h & 0x8000 ? -v : v;
}

template <typename T> struct Nd { static const int v = 7; };
template <> struct Nd<float> { static const int v = 4; };
static long double lval(double x) { return x; }
static long double lval(float x) { return x; }

template <typename T> static T make(double x) { return T(x); }

template <typename T>
static void check(const char *name, int n, double ds, double L, int spread) {
  const int nd = Nd<T>::v, H = n / 2, kg = (H + 15) / 16, NB = 4 * kg - 1;
  std::vector<double> g(n);
  for (int m = 0; m < n; ++m) {
    const double k = 2 * 3.1415926535 * (m <= n / 2 - 1 ? m : m - n) / L;
    g[m] = exp(-ds * k * k) / n;
  }
  std::vector<unsigned char> tab;
  if (!tc_build_table(g.data(), n, nd, tab, nullptr)) {
    printf("%s %d no-table 0\n", name, n);
    return;
  }
  const int *head = reinterpret_cast<const int *>(tab.data());
  const uint16_t *dig = reinterpret_cast<const uint16_t *>(tab.data() + 16);
  auto bdig = [&](int par, int j, int row, int k) {   // as the descriptors address it
    const uint16_t *half = dig + (size_t)par * tc::b_half_bytes(nd, kg) / 2;
    const int gc = tc::group_cols(nd, kg), rounds = tc::split_rows(nd, kg) ? 2 : 1;
    const int rd = rounds == 2 ? row / 8 % 2 : 0, col = rounds == 2 ? row / 16 * 8 + row % 8 : row;
    const int r = (rd * nd + j) * gc + col, blk = row / 8 + (2 * kg - 1) - k / 8;
    const size_t core = tc::dense_b(kg) ? (size_t)(k / 8) * (rounds * nd * gc / 8) + r / 8
                                        : (size_t)j * NB + blk;
    return f16(half[core * 64 + (row % 8) * 8 + k % 8]);
  };
  std::vector<long double> K(n, 0.0L);
  const long double tp = 6.283185307179586476925286766559L;
  for (int d = 0; d < n; ++d)
    for (int m = 0; m < n; ++m) K[d] += (long double)g[m] * cosl(tp * ((long long)m * d % n) / n);
  double worst = 0.0, maxacc = 0.0;
  srand(n);
  for (int rep = 0; rep < 20; ++rep) {
    std::vector<T> x(n);
    for (int i = 0; i < n; ++i) {
      double r = rand() / (double)RAND_MAX + rand() / (double)RAND_MAX / RAND_MAX;
      if (rep % 4 == 1) r = r - 0.5;
      if (rep % 4 == 2) r = ldexp(r, -(rand() % (spread + 1)));
      if (rep % 4 == 3) r = 1.0 + 1e-3 * r;
      x[i] = make<T>(r * (rep % 5 == 0 ? 1e-12 : 3.7));
    }
    int key = 0;
    for (int i = 0; i < n; ++i) key = mag_key(x[i]) > key ? mag_key(x[i]) : key;
    const int E = line_exp(T(0.0f), key);
    std::vector<long long> c[2];
    for (int k = 0; k < H; ++k) {
      const long long a = to_fixed(x[k], E), b = to_fixed(x[k + H], E);
      c[0].push_back(a + b);
      c[1].push_back(a - b);
    }
    std::vector<double> acc[2];
    std::vector<long long> yi[2];
    std::vector<float> yf[2];
    for (int par = 0; par < 2; ++par)
      for (int row = 0; row < H; ++row) {
        double D[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int k = 0; k < H; ++k) {
          const unsigned long long z = nd == 7 ? biased_digits((int64_t)c[par][k])
                                               : biased_digits((int)c[par][k]);
          for (int i = 0; i < nd; ++i) {
            const int d = (int)((z >> (8 * (nd - 1 - i))) & (i == 0 ? 0xffff : 0xff)) - 128;
            for (int j = 0; i + j < nd; ++j) D[i + j] += d * bdig(par, j, row, k);
          }
        }
        for (int q = 0; q < nd; ++q) maxacc = fabs(D[q]) > maxacc ? fabs(D[q]) : maxacc;
        if (nd == 7) {
          long long s = ((long long)D[0] * 256 + (long long)D[1]) << 32;
          s += ((long long)D[2] * 256 + (long long)D[3]) * 65536;
          s += (long long)D[4] * 256 + (long long)D[5] + (((long long)D[6] + 128) >> 8);
          yi[par].push_back(s);
        } else {
          yf[par].push_back(fmaf(fmaf(fmaf((float)D[0], 256.f, (float)D[1]), 256.f, (float)D[2]),
                                 256.f, (float)D[3]));
        }
      }
    const int ue = unit_exp(T(0.0f), E) + (nd == 7 ? 55 : 23) - head[0];
    long double mx = 0.0L;
    for (int i = 0; i < n; ++i) mx = fabsl(lval(x[i])) > mx ? fabsl(lval(x[i])) : mx;
    for (int i = 0; i < n; ++i) {
      long double ref = 0.0L;
      for (int k = 0; k < n; ++k) ref += K[(i - k + n) % n] * lval(x[k]);
      const int m = i % H;
      long double y;
      if constexpr (nd == 7)
        y = lval(from_fixed(i < H ? yi[0][m] + yi[1][m] : yi[0][m] - yi[1][m], ue, T()));
      else
        y = scale2(i < H ? yf[0][m] + yf[1][m] : yf[0][m] - yf[1][m], ue);
      const double e = (double)(fabsl(y - ref) / mx);
      worst = e > worst ? e : worst;
    }
  }
  printf("%s %d %.3g %.0f\n", name, n, worst, maxacc);
}

int main() {
  const int ns[] = {2, 6, 16, 24, 32, 50, 64, 96, 100, 126, 128};
  for (int n : ns) {
    check<double>("f64", n, 0.01, 4.0, 40);
    check<float>("f32", n, 0.005, 3.8, 20);
    check<double>("f64wide", n, 1.0, 3.0, 40);     // a kernel as wide as the box
    check<double>("f64narrow", n, 1e-4, 9.0, 40);  // ripples of both signs
  }
  check<float>("f32", 160, 0.005, 5.0, 20);
  check<float>("f32", 256, 0.005, 8.0, 20);
  return 0;
}
