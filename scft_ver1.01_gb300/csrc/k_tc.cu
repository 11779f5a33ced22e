// Tensor-core passes of the propagator march (core and arithmetic: tc_core.cuh).
//
// k_real: one axis pass on working reals, out = post * K (pre * in), and for
// FP32 the fused step pair.  k_fix: the fused march of FP64 contexts,
// whose intermediates between passes stay 64-bit integers, so that a pass costs no
// conversion to or from the working real (those were about half of a pass's 142
// instructions per point):
//   first  v0 = W q0 and the first filter        real in, integers out
//   mid    one filter                            integers in and out
//   pair   filter, q = W y (stored), v = W q, filter
//   last   filter, q = W y (stored)              integers in, real out
// A filtered line goes out as it comes from the products, its unit (a power of two,
// 16 bits) into an array by lines; the next pass, along another axis, gives every
// point the unit of the line that it came from, and rescales its own lines to the
// digits' 2^54 by their largest value.  So a line keeps the accuracy of its own scale
// wherever in the instance it lies, as with reals, and exponents have no range to
// leave.  (One unit for an instance and step, from bounds, is about 10 % faster, 64^3 3.53
// ms per SCF iteration with 200 steps against 3.83, but values far below the largest lose
// their last bits to it: beside a well 4e-10 off where FFTs leave 2e-11.)
#include "tc_core.cuh"

#include <limits.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

namespace scft {

namespace {

using namespace tc;

template <typename T> constexpr int kNd = 7;
template <> constexpr int kNd<float> = 4;

__device__ __forceinline__ double bad_value(double) { return __longlong_as_double(0x7ff8000000000000LL); }
__device__ __forceinline__ float bad_value(float) { return __int_as_float(0x7fc00000); }

// filter result -> working real (float: y * 2^ue)
template <typename T, typename A> __device__ __forceinline__ T finish_real(A y, int ue) {
  if constexpr (std::is_same<T, float>::value) return scale2(y, ue);
  else return from_fixed(y, ue, T());
}

// Geometry of a pass's lines.
struct Lines {
  Shape sh;
  int n;
  long long lines;       // per instance
  long long row_len;     // column passes: consecutive lines of one row
  long long s_outer, s_n;
};

// f(row, column, offset in the tile) over the tile's contiguous rows by the nt
// computing threads, coalesced
template <typename F> __device__ __forceinline__ void over_rows(int nt, int n, int nl, F &&f) {
  int r = (int)threadIdx.x / n, col = (int)threadIdx.x % n;
  const int dr = nt / n, dc = nt % n;
  for (int i = threadIdx.x; i < nl * n; i += nt) {
    f(r, col, i);
    r += dr;
    col += dc;
    if (col >= n) {
      col -= n;
      ++r;
    }
  }
}

// f(row, column, offset, load(offset)) with U loads in flight per thread.  One at a
// time the FP32 x passes waited for them (100 x 80 x 60: 26 us where a column pass
// takes 10; 4.8 ms per SCF iteration, with 8 in flight 4.3).  64-bit values take 4:
// 8 were no faster (96^3 9.7 against 9.4 ms) and spilled.
template <int U, typename L, typename F>
__device__ __forceinline__ void over_rows(int nt, int n, int nl, L &&load, F &&f) {
  typedef decltype(load(0)) V;
  const int total = nl * n;
  int r = (int)threadIdx.x / n, col = (int)threadIdx.x % n;
  const int dr = nt / n, dc = nt % n;
#pragma unroll 1
  for (int i0 = threadIdx.x; i0 < total; i0 += U * nt) {
    V x[U];
#pragma unroll
    for (int j = 0; j < U; ++j) x[j] = i0 + j * nt < total ? load(i0 + j * nt) : V();
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (i0 + j * nt < total) f(r, col, i0 + j * nt, x[j]);
      r += dr;
      col += dc;
      if (col >= n) {
        col -= n;
        ++r;
      }
    }
  }
}
template <typename T> struct WithFactor {
  T x, w;
};

// ------------------------------------------------------------------ k_real
template <typename T, int MAXT, int PP, bool XP, bool PAIR>
__global__ void __launch_bounds__(MAXT, 1) k_real(Lines ln, const void *table_, PassSet<T, kStepSet> ps) {
  typedef Tile<kNd<T>, PP> E;
  typedef typename E::I I;
  typedef typename E::Acc Acc;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  E e;
  const void *table = table_;
  if constexpr (std::is_same<T, float>::value) {
    if (ps.desc) table = ps.desc[blockIdx.z].tc;
  }
  e.setup(smem_raw, ln.sh, table, table);
  const TcHead head = *static_cast<const TcHead *>(table);
  const int set = set_of(ps);
  const long long b = (long long)blockIdx.z - (long long)set * ps.batch;
  const long long line0 = (long long)blockIdx.x * e.ln;
  const int nl = (int)min((long long)e.ln, ln.lines - line0);
  const T *in = ps.in[set] + b * ps.in_bs[set];
  T *out = ps.out[set] + b * ps.out_bs[set];
  const T *pre = ps.pre[set] ? ps.pre[set] + b * ps.w_bs : nullptr;
  const T *post = ps.post[set] ? ps.post[set] + b * ps.w_bs : nullptr;
  T *qo = PAIR ? ps.qout[set] + b * ps.qout_bs[set] : nullptr;
  if constexpr (std::is_same<T, float>::value && !PAIR) {
    if (ps.desc) {   // a batched pass: this line set's own buffers
      const PassDesc d = ps.desc[blockIdx.z];
      in = d.in;
      out = d.out;
      pre = d.pre;
      post = d.post;
    }
  }
  const int H = ln.sh.half[0];
  pdl_wait();      // the input is the previous pass's output
  pdl_release();
  if (e.issuer) {
    e.run_issuer(PAIR ? 2 : 1, [](int) { return 0; });
    e.finish(ps.err);
    return;
  }
  e.run_compute();
  const bool mine = e.line < nl;
  const long long c = line0 + e.line;
  const long long base = XP ? 0 : (mine ? (c / ln.row_len) * ln.s_outer + c % ln.row_len : 0);
  const long long tile = XP ? line0 * ln.n : 0;   // x pass: contiguous rows
  const int P = ln.n + 1;                         // staging pitch
  T *stg = reinterpret_cast<T *>(smem_raw);

  T a[PP], bb[PP];
  if constexpr (XP) {
    const T *src = in + tile, *wsrc = pre ? pre + tile : nullptr;
    constexpr int U = sizeof(T) == 4 ? 8 : 4;
    if (wsrc)
      over_rows<U>(e.ncomp, ln.n, nl, [&](int i) { return WithFactor<T>{ldg(src + i), ldg(wsrc + i)}; },
                   [&](int r, int col, int, WithFactor<T> v) { stg[r * P + col] = v.x * v.w; });
    else
      over_rows<U>(e.ncomp, ln.n, nl, [&](int i) { return ldg(src + i); },
                   [&](int r, int col, int, T x) { stg[r * P + col] = x; });
    e.sync();
  }
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    const int k = PP * e.blk + i;
    a[i] = bb[i] = T(0.0f);
    if (mine && k < H) {
      if constexpr (XP) {
        a[i] = stg[e.line * P + k];
        bb[i] = stg[e.line * P + k + H];
      } else {
        a[i] = ldg(in + base + (long long)k * ln.s_n);
        bb[i] = ldg(in + base + (long long)(k + H) * ln.s_n);
      }
    }
  }
  if constexpr (!XP) {
    if (pre) {
#pragma unroll
      for (int i = 0; i < PP; ++i) {
        const int k = PP * e.blk + i;
        if (mine && k < H) {
          a[i] = a[i] * ldg(pre + base + (long long)k * ln.s_n);
          bb[i] = bb[i] * ldg(pre + base + (long long)(k + H) * ln.s_n);
        }
      }
    }
  }
  int key = 0;
#pragma unroll
  for (int i = 0; i < PP; ++i) key = max(key, max(mag_key(a[i]), mag_key(bb[i])));
  e.start();   // TMEM address, cleared keys; the staging tile is read
  key = e.line_key(0, key);
  bool bad = key >= bad_key<T>();
  int Eb = line_exp(T(0.0f), key);
  I xa[PP], xb[PP];
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    xa[i] = to_fixed(a[i], Eb);
    xb[i] = to_fixed(bb[i], Eb);
  }
  // results come in units of 2^(unit + shift)
  const int shift = (kNd<T> == 7 ? 55 - kFine : 23) - head.kshift;
  int ue = unit_exp(T(0.0f), Eb) + shift;

  if constexpr (PAIR) {
    T ya[PP], yb[PP];
    e.filter(xa, xb, []() {}, [&](int i, Acc p, Acc q) {
      ya[i] = bad ? bad_value(T(0.0f)) : finish_real<T>(p, ue);
      yb[i] = bad ? bad_value(T(0.0f)) : finish_real<T>(q, ue);
    });
    if constexpr (XP) {
      e.sync();
#pragma unroll
      for (int i = 0; i < PP; ++i) {
        const int k = PP * e.blk + i;
        if (mine && k < H) {
          stg[e.line * P + k] = ya[i];
          stg[e.line * P + k + H] = yb[i];
        }
      }
      e.sync();
      over_rows<8>(e.ncomp, ln.n, nl, [&](int i) { return ldg(post + tile + i); },
                   [&](int r, int col, int i, T w) {
        const T q = stg[r * P + col] * w;
        qo[tile + i] = q;
        stg[r * P + col] = q * w;
      });
      e.sync();
#pragma unroll
      for (int i = 0; i < PP; ++i) {
        const int k = PP * e.blk + i;
        const bool on = mine && k < H;
        ya[i] = on ? stg[e.line * P + k] : T(0.0f);
        yb[i] = on ? stg[e.line * P + k + H] : T(0.0f);
      }
    } else {
      if constexpr (MAXT > 640) {   // 64 registers: no room for loads ahead
#pragma unroll
        for (int i = 0; i < PP; ++i) {
          const int k = PP * e.blk + i;
          if (mine && k < H) {
            const long long o0 = base + (long long)k * ln.s_n, o1 = o0 + (long long)H * ln.s_n;
            const T w0 = ldg(post + o0), w1 = ldg(post + o1);
            const T q0 = ya[i] * w0, q1 = yb[i] * w1;
            qo[o0] = q0;
            qo[o1] = q1;
            ya[i] = q0 * w0;
            yb[i] = q1 * w1;
          } else {
            ya[i] = yb[i] = T(0.0f);
          }
        }
      } else {
        // loads of four points first: behind a branch each they waited one by one (60^3
        // 2.23 -> 2.14 ms per SCF iteration; 1024 threads spilled: 40 x 36 x 160 3.95 -> 4.17)
#pragma unroll
        for (int g = 0; g < PP; g += 4) {
          T w0[4], w1[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int k = PP * e.blk + g + i;
            const long long o0 = base + (long long)k * ln.s_n;
            w0[i] = mine && k < H ? ldg(post + o0) : T(0.0f);
            w1[i] = mine && k < H ? ldg(post + o0 + (long long)H * ln.s_n) : T(0.0f);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int k = PP * e.blk + g + i;
            const bool on = mine && k < H;
            const long long o0 = base + (long long)k * ln.s_n;
            const T q0 = ya[g + i] * w0[i], q1 = yb[g + i] * w1[i];
            if (on) {
              qo[o0] = q0;
              qo[o0 + (long long)H * ln.s_n] = q1;
            }
            ya[g + i] = on ? q0 * w0[i] : T(0.0f);
            yb[g + i] = on ? q1 * w1[i] : T(0.0f);
          }
        }
      }
    }
    int key2 = 0;
#pragma unroll
    for (int i = 0; i < PP; ++i) key2 = max(key2, max(mag_key(ya[i]), mag_key(yb[i])));
    key2 = e.line_key(1, key2);   // (its barrier: the staging tile is read)
    bad = key2 >= bad_key<T>();
    Eb = line_exp(T(0.0f), key2);
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      xa[i] = to_fixed(ya[i], Eb);
      xb[i] = to_fixed(yb[i], Eb);
    }
    ue = unit_exp(T(0.0f), Eb) + shift;
  }

  if constexpr (XP) {
    // row by row through the staging tile (A is free once the products are done)
    T ya[PP], yb[PP];
    e.filter(xa, xb, []() {}, [&](int i, Acc p, Acc q) {
      ya[i] = bad ? bad_value(T(0.0f)) : finish_real<T>(p, ue);
      yb[i] = bad ? bad_value(T(0.0f)) : finish_real<T>(q, ue);
    });
    e.sync();
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      const int k = PP * e.blk + i;
      if (mine && k < H) {
        stg[e.line * P + k] = ya[i];
        stg[e.line * P + k + H] = yb[i];
      }
    }
    e.sync();
    const T *wd = !PAIR && post ? post + tile : nullptr;
    if (wd)
      over_rows<4>(e.ncomp, ln.n, nl, [&](int i) { return ldg(wd + i); },
                   [&](int r, int col, int i, T w) { out[tile + i] = stg[r * P + col] * w; });
    else
      over_rows(e.ncomp, ln.n, nl, [&](int r, int col, int i) { out[tile + i] = stg[r * P + col]; });
  } else {
    e.filter(xa, xb, []() {}, [&](int i, Acc p, Acc q) {
      const int k = PP * e.blk + i;
      if (mine && k < H) {
        const long long o0 = base + (long long)k * ln.s_n, o1 = o0 + (long long)H * ln.s_n;
        T r0 = bad ? bad_value(T(0.0f)) : finish_real<T>(p, ue);
        T r1 = bad ? bad_value(T(0.0f)) : finish_real<T>(q, ue);
        if (!PAIR && post) {
          r0 = r0 * ldg(post + o0);
          r1 = r1 * ldg(post + o1);
        }
        out[o0] = r0;
        out[o1] = r1;
      }
    });
  }
  e.finish(ps.err);
}

// ------------------------------------------------------------------ k_fix
enum { FIRST = 0, MID = 1, PAIR = 2, LAST = 3 };

// Units lie within +-5300 (values that are neither infinite nor 0 as reals, line_unit).
// That of a line whose values are not finite: of its points, and what its integers are
// rescaled to.
constexpr int kBadUnit = 0x7fff, kBadLine = 1 << 21, kKeyBias = 1 << 22;

__device__ __forceinline__ int64_t ld64(const int64_t *p) {
  return __ldg(reinterpret_cast<const long long *>(p));
}
__device__ __forceinline__ uint64_t ldw(const double *p) {
  return (uint64_t)__ldg(reinterpret_cast<const long long *>(p));
}
// A point's exponent bound (|x| * 2^u <= 2^e) as a key of its line, and the unit of a
// line's integers, |X| <= 2^54, from its largest key.  With 55 bits for every point that
// unit is above all of theirs: they are only shifted to the right (7 instructions a point
// instead of 12), and what that rounds off is below the rounding that the point of the
// largest unit brings along.  Values of 2^1024 and more are infinite as reals; below
// 2^-1100 they are 0.
__device__ __forceinline__ int point_key(int64_t x, int u) { return u + bits_of(x) + kKeyBias; }
__device__ __forceinline__ int line_unit(int key) {
  const int e = max(key - kKeyBias, -1100);
  return e > 1024 ? kBadLine : e - 54;
}
__device__ __forceinline__ int16_t short_unit(int u) { return (int16_t)min(u, kBadUnit); }
// r * 2^ur as the stored slice's value
__device__ __forceinline__ double slice_value(int64_t r, int ur) {
  const int h = (int)(r >> 32);
  if (h != (h >> 31) && fast_units(ur)) return from_fixed_fast(r, ur);
  return ur >= kBadUnit / 2 ? bad_value(0.0) : from_fixed(r, ur, 0.0);
}
__device__ __forceinline__ Factor any_factor(uint64_t w) {
  return factor_rare(w) ? factor_of_rare(w) : factor_of(w);
}
// The units of a thread's points, until their line's is known: two 16-bit numbers in a
// register.
template <int PP> struct Units {
  uint32_t v[PP];
  __device__ __forceinline__ void set(int i, int u0, int u1) {
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(v[i]) : "r"(u1), "r"(u0));
  }
  __device__ __forceinline__ int a(int i) const { return (int16_t)v[i]; }
  __device__ __forceinline__ int b(int i) const { return (int)v[i] >> 16; }
};
// A thread's points of a column line: PP at off, off + sn, ..., and as many
// another hs on; the first `lim` exist.
struct Column {
  unsigned off, sn, hs;
  int lim;
};
// q = W y to the finished slice and x = W q, in units of 2^u, for N/2 points (x[2j]: y of
// point g + j of the column in units of 2^uo, x[2j + 1]: of its partner); returns the
// largest key.  Without a branch in it, so that the N chains (about 190 cycles each) run
// side by side: factors that are not normal numbers are set right before, values that
// the fast conversion does not take are stored again afterwards.
template <int N>
__device__ __forceinline__ int factor_group(int64_t (&x)[N], int (&u)[N], const double *w, double *qo,
                                            const Column &c, int g, int uo) {
  auto at = [&](int i) { return c.off + (g + i / 2) * c.sn + (i & 1) * c.hs; };
  uint64_t b[N];
  Factor f[N];
  bool rare = false, slow = (uint32_t)(uo + 490) >= 880u;   // (then ur is a fast unit)
#pragma unroll
  for (int i = 0; i < N; ++i) b[i] = g + i / 2 < c.lim ? ldw(w + at(i)) : 0x3ff0000000000000ULL;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    rare |= factor_rare(b[i]);
    f[i] = factor_of(b[i]);
  }
  if (rare) {
    slow = true;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (factor_rare(b[i])) f[i] = factor_of_rare(b[i]);
  }
  int64_t r[N];
  int key = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    r[i] = mul_w62(x[i], f[i]);
    const int ur = uo + f[i].e - 1022, h = (int)(r[i] >> 32);
    const bool on = g + i / 2 < c.lim;
    slow |= on && h == (h >> 31);
    const double q = from_fixed_fast(r[i], ur);
    if (on) qo[at(i)] = q;
    x[i] = mul_w62(r[i], f[i]);
    u[i] = ur + f[i].e - 1022;
    key = max(key, on ? point_key(x[i], u[i]) : 0);
  }
  if (slow) {
#pragma unroll 1
    for (int i = 0; i < N; ++i) {
      int64_t ri = r[0];
      int ui = f[0].e;
#pragma unroll
      for (int j = 1; j < N; ++j) {
        ri = i == j ? r[j] : ri;
        ui = i == j ? f[j].e : ui;
      }
      if (g + i / 2 < c.lim) qo[at(i)] = slice_value(ri, uo + ui - 1022);
    }
  }
  return key;
}
// The same for all of a thread's points.
template <int PP>
__device__ __forceinline__ int factor_points(int64_t (&xa)[PP], int64_t (&xb)[PP], Units<PP> &un,
                                             const double *w, double *qo, const Column &c, int uo) {
  int key = 0;
#pragma unroll
  for (int g = 0; g < PP; g += 4) {
    int64_t x[8];
    int u[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[2 * i] = xa[g + i];
      x[2 * i + 1] = xb[g + i];
    }
    key = max(key, factor_group(x, u, w, qo, c, g, uo));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      xa[g + i] = x[2 * i];
      xb[g + i] = x[2 * i + 1];
      un.set(g + i, u[2 * i], u[2 * i + 1]);
    }
  }
  return key;
}
// A thread's points (16 and their partners) in the staging memory, where they
// cost no registers: as unrolled code over registers the factor step of 16
// points spilled 560-800 bytes a thread.
struct Staged {
  int64_t *own;
  int16_t *units;
  int stride;
  __device__ __forceinline__ int64_t &a(int i) const { return own[2 * i * stride]; }
  __device__ __forceinline__ int64_t &b(int i) const { return own[(2 * i + 1) * stride]; }
  __device__ __forceinline__ int ua(int i) const { return units[2 * i * stride]; }
  __device__ __forceinline__ int ub(int i) const { return units[(2 * i + 1) * stride]; }
  __device__ __forceinline__ int factor(const double *w, double *qo, const Column &c, int uo) const {
    int key = 0;
#pragma unroll 1
    for (int g = 0; g < 16; g += 4) {
      int64_t x[8];
      int u[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[2 * i] = a(g + i);
        x[2 * i + 1] = b(g + i);
      }
      key = max(key, factor_group(x, u, w, qo, c, g, uo));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a(g + i) = x[2 * i];
        b(g + i) = x[2 * i + 1];
        units[2 * (g + i) * stride] = short_unit(u[2 * i]);
        units[(2 * (g + i) + 1) * stride] = short_unit(u[2 * i + 1]);
      }
    }
    return key;
  }
};

// v0 = W q0 for all of a thread's points, as factor_group does it.
template <int PP>
__device__ __forceinline__ int first_points(int64_t (&xa)[PP], int64_t (&xb)[PP], Units<PP> &un,
                                            const double *in, const double *w, const Column &c) {
  int key = 0;
#pragma unroll
  for (int g = 0; g < PP; g += 2) {
    uint64_t b[4], q[4];
    Factor f[4];
    int64_t x[4];
    int u[4];
    bool rare = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned o = c.off + (g + i / 2) * c.sn + (i & 1) * c.hs;
      const bool on = g + i / 2 < c.lim;
      b[i] = on ? ldw(w + o) : 0x3ff0000000000000ULL;
      q[i] = on ? ldw(in + o) : 0x3ff0000000000000ULL;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      rare |= factor_rare(b[i]) || real_rare(q[i]);
      f[i] = factor_of(b[i]);
      x[i] = split_real(q[i], u[i]);
    }
    if (rare) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        f[i] = any_factor(b[i]);
        if (real_rare(q[i])) x[i] = split_real_rare(q[i], u[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool on = g + i / 2 < c.lim;
      x[i] = on ? mul_w62(x[i], f[i]) : 0;
      u[i] += f[i].e - 1022;
      key = max(key, on ? point_key(x[i], u[i]) : 0);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      xa[g + j] = x[2 * j];
      xb[g + j] = x[2 * j + 1];
      un.set(g + j, u[2 * j], u[2 * j + 1]);
    }
  }
  return key;
}
// A thread's points, x(i, half) in units of 2^u(i, half), and their largest key.  Units
// first: with 16 points the registers do not hold the loads of both at once, and units
// behind the points came in several rounds of their own.
template <int PP, typename X, typename U>
__device__ __forceinline__ int load_points(int64_t (&xa)[PP], int64_t (&xb)[PP], Units<PP> &un, int lim,
                                           X &&x, U &&u) {
  int key = 0;
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    int u0 = 0, u1 = 0;
    if (i < lim) {
      u0 = u(i, 0);
      u1 = u(i, 1);
    }
    un.set(i, u0, u1);
  }
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    xa[i] = i < lim ? x(i, 0) : 0;
    xb[i] = i < lim ? x(i, 1) : 0;
  }
#pragma unroll
  for (int i = 0; i < PP; ++i)
    if (i < lim) key = max(key, max(point_key(xa[i], un.a(i)), point_key(xb[i], un.b(i))));
  return key;
}
// ... to the unit of their line.
template <int PP>
__device__ __forceinline__ void scale_points(int64_t (&xa)[PP], int64_t (&xb)[PP], const Units<PP> &un,
                                             int ue) {
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    xa[i] = shifted(xa[i], ue - un.a(i));
    xb[i] = shifted(xb[i], ue - un.b(i));
  }
}

template <int PP, bool XP, int MODE>
__global__ void __launch_bounds__(PP == 16 ? 640 : 544, 1) k_fix(Lines ln, const void *table, FixPass fp) {
  typedef Tile<7, PP> E;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  E e;
  e.setup(smem_raw, ln.sh, table, table);
  const TcHead head = *static_cast<const TcHead *>(table);
  const long long b = blockIdx.z;
  const unsigned line0 = blockIdx.x * e.ln;
  const int nl = (int)min((long long)e.ln, ln.lines - line0);
  const unsigned H = ln.sh.half[0];
  pdl_wait();      // the input is the previous pass's output
  pdl_release();
  if (e.issuer) {
    e.run_issuer(MODE == PAIR ? 2 : 1, [](int) { return 0; });
    e.finish(fp.err);
    return;
  }
  e.run_compute();
  // element offsets within an instance fit 32 bits (lines of at most 128 points)
  const unsigned c = line0 + e.line, rl = (unsigned)ln.row_len;
  const unsigned base = XP ? c * ln.n : (c / rl) * (unsigned)ln.s_outer + c % rl;
  const unsigned sn = XP ? 1 : (unsigned)ln.s_n;
  const unsigned k0 = PP * e.blk, tile = line0 * ln.n;
  const unsigned off = base + k0 * sn, hs = H * sn;
  const int lim = e.line < nl ? (int)H - (int)k0 : 0;   // this thread's points: i < lim
  const Column col{off, sn, hs, lim};
  const int P = ln.n + 1;
  int64_t *stg = reinterpret_cast<int64_t *>(smem_raw);
  int64_t *row = stg + e.line * P + k0;                 // its points in the staging tile
  int *ur_row = reinterpret_cast<int *>(smem_raw + e.lay.ur_off);
  int16_t *us = reinterpret_cast<int16_t *>(smem_raw + ln.sh.units_off);
  int16_t *urow = us + e.line * P + k0;                 // rows' units, as the points lie
  const double *w = fp.w + b * fp.w_bs;
  const int shift = 55 - kFine - head.kshift;

  int64_t xa[PP], xb[PP];
  Units<PP> un;
  int key = 0;
  if constexpr (MODE == FIRST) {
    // real slice times the factor; a handful of launches per iteration, so the
    // x pass reads its rows without staging
    key = first_points(xa, xb, un, static_cast<const double *>(fp.in) + b * fp.in_bs, w, col);
  } else {
    const int64_t *in = static_cast<const int64_t *>(fp.in) + b * fp.in_bs;
    if constexpr (XP) {
      over_rows<4>(e.ncomp, ln.n, nl, [&](int i) { return ld64(in + tile + i); },
                   [&](int r, int cc, int, int64_t x) { stg[r * P + cc] = x; });
      e.sync();
    }
    const int16_t *u_in = fp.u_in + b * fp.u_in_bs + (c / fp.u_div) * fp.u_quo + (c % fp.u_div) * fp.u_rem +
                      k0 * fp.u_step;
    key = load_points(
        xa, xb, un, lim,
        [&](int i, int half) { return XP ? row[i + half * H] : ld64(in + (off + i * sn + half * hs)); },
        [&](int i, int half) { return (int)__ldg(u_in + (i + half * H) * fp.u_step); });
  }
  e.start();   // TMEM address, cleared keys; the staging tile is read

  // The filters and what follows each.  One copy of the code serves both
  // filters of a pair: with two a pair was 7450 instructions long (119 KB at
  // N = 128) and waited for them.
  int64_t *out = static_cast<int64_t *>(fp.out) + b * fp.out_bs;
  constexpr bool kStaged = PP == 16 && !XP && (MODE == PAIR || MODE == LAST);
  const Staged sp{stg + threadIdx.x, us + threadIdx.x, e.ncomp};
  int uo = 0;                   // the unit of the filtered line
#pragma unroll 1
  for (int f = 0; f < (MODE == PAIR ? 2 : 1); ++f) {
    key = e.line_key(f, key);   // (its barrier: the staging tile is read)
    const int ue = line_unit(key);
    scale_points(xa, xb, un, ue);
    if constexpr (kStaged) {
      e.filter(xa, xb, []() {}, [&](int i, int64_t p, int64_t q) {
        if (i < 8) {
          xa[i] = p;
          xb[i] = q;
        } else {   // the last products are done: A is free
          sp.a(i) = p;
          sp.b(i) = q;
        }
      });
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        sp.a(i) = xa[i];
        sp.b(i) = xb[i];
      }
    } else {
      e.filter(xa, xb, []() {});
    }
    uo = ue == kBadLine ? kBadUnit : ue + shift;
    if (MODE == LAST || (MODE == PAIR && f == 0)) {
      double *qo = static_cast<double *>(fp.q) + b * fp.q_bs;
      if constexpr (XP) {
        e.sync();   // A is free
        if (e.blk == 0) ur_row[e.line] = uo;
#pragma unroll
        for (int i = 0; i < PP; ++i) {
          if (i < lim) {
            row[i] = xa[i];
            row[i + H] = xb[i];
          }
        }
        e.sync();
        over_rows<4>(e.ncomp, ln.n, nl, [&](int i) { return ldw(w + tile + i); },
                     [&](int r, int cc, int i, uint64_t wb) {
          const Factor fa = any_factor(wb);
          const int ur = ur_row[r] + fa.e - 1022;
          const int64_t v = mul_w62(stg[r * P + cc], fa);
          qo[tile + i] = slice_value(v, ur);
          if (MODE == PAIR) {
            stg[r * P + cc] = mul_w62(v, fa);
            us[r * P + cc] = short_unit(ur + fa.e - 1022);
          }
        });
        if constexpr (MODE == PAIR) {
          e.sync();
          key = 0;
#pragma unroll
          for (int i = 0; i < PP; ++i) {
            xa[i] = xb[i] = 0;
            if (i < lim) {
              xa[i] = row[i];
              xb[i] = row[i + H];
              const int u0 = urow[i], u1 = urow[i + H];
              un.set(i, u0, u1);
              key = max(key, max(point_key(xa[i], u0), point_key(xb[i], u1)));
            }
          }
        }
      } else if constexpr (kStaged) {
        key = sp.factor(w, qo, col, uo);
#pragma unroll
        for (int i = 0; i < PP && MODE == PAIR; ++i) {
          xa[i] = sp.a(i);
          xb[i] = sp.b(i);
          un.set(i, sp.ua(i), sp.ub(i));
        }
      } else if constexpr (PP <= 8) {
        key = factor_points(xa, xb, un, w, qo, col, uo);
      }
    }
  }

  if constexpr (MODE != LAST) {
    if (e.blk == 0 && e.line < nl) fp.u_out[b * fp.u_out_bs + c] = (int16_t)uo;
    if constexpr (XP) {
      e.sync();   // A is free
#pragma unroll
      for (int i = 0; i < PP; ++i) {
        if (i < lim) {
          row[i] = xa[i];
          row[i + H] = xb[i];
        }
      }
      e.sync();
      over_rows(e.ncomp, ln.n, nl, [&](int r, int cc, int i) { out[tile + i] = stg[r * P + cc]; });
    } else if constexpr (kStaged) {
#pragma unroll 4
      for (int i = 0; i < PP; ++i) {
        if (i < lim) {
          out[off + i * sn] = sp.a(i);
          out[off + i * sn + hs] = sp.b(i);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < PP; ++i) {
        if (i < lim) {
          out[off + i * sn] = xa[i];
          out[off + i * sn + hs] = xb[i];
        }
      }
    }
  }
  e.finish(fp.err);
}

// ---------------------------------------------------------------- k_planes
// Whole planes per CTA (up to 64 points a line): both axes of a step in one
// launch.  What a launch costs beside its filters (2.7 us until the next one may
// read, 1.5 us to load and store a tile) was about half of a 64^3 step.  ms per
// SCF iteration with 200 steps, one launch per pass against planes: FP64 32^3 2.54 /
// 2.17, 64^3 4.22 / 3.81.  Above 64 points the planes' one CTA each takes as long as the
// passes' more evenly filled ones (with one unit per instance: 128^3 22.5 / 22.4, 96^3
// 10.1 / 12.3; FP32 80^3 5.4 / 6.2): those keep their passes.
//
// FILM false: x filter, y filter, q = W y (stored), v = W q, y filter, x filter
// (the middle pass, the pair and the next middle pass of k_fix's schedule).
// FILM true (nz = 1): a whole march segment, step after step, in one launch of
// one CTA per instance: nothing of a film leaves the CTA but its slices.
//
// Between its filters the planes lie in shared memory as integers of their lines'
// units (rows of nx + 1: conflict-free along both axes).  q and W are read and written
// from the y lines, where consecutive lines are consecutive in memory.
struct PlaneArgs {
  Shape sh;
  int nx, ny, nz, per;   // per: planes per CTA
  int steps;             // FILM: contour steps of the segment
  long long q_step;      // FILM: from one slice to the next
};
template <int PP, bool FILM>
__global__ void __launch_bounds__(544, 1)
    k_planes(PlaneArgs pa, const void *tx, const void *ty, FixPass fp) {
  typedef Tile<7, PP> E;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  E e;
  e.setup(smem_raw, pa.sh, tx, ty);
  const int shift_x = 55 - kFine - static_cast<const TcHead *>(tx)->kshift;
  const int shift_y = 55 - kFine - static_cast<const TcHead *>(ty)->kshift;
  const long long b = blockIdx.z;
  const int filters = FILM ? 2 * pa.steps : 4;
  auto axis_of = [](int f) { return FILM ? f & 1 : (f == 1 || f == 2 ? 1 : 0); };
  pdl_wait();
  pdl_release();
  if (e.issuer) {
    e.run_issuer(filters, axis_of);
    e.finish(fp.err);
    return;
  }
  e.run_compute();
  const int nx = pa.nx, ny = pa.ny, P = nx + 1;
  const int z0 = blockIdx.x * pa.per, np = min(pa.per, pa.nz - z0);
  const unsigned tile = (unsigned)z0 * ny * nx;
  const int k0 = PP * e.blk, pl = e.line / nx, xx = e.line - pl * nx;
  int64_t *S = reinterpret_cast<int64_t *>(smem_raw);
  // units: of the lines last filtered along each axis, and of points that have their own
  int16_t *ul = reinterpret_cast<int16_t *>(smem_raw + e.lay.ur_off);
  int16_t *us = reinterpret_cast<int16_t *>(smem_raw + pa.sh.units_off);
  const double *w = fp.w + b * fp.w_bs;
  // this thread's points as x line (row `line`) and as y line (plane pl, x)
  const int lim_x = e.line < np * ny ? pa.sh.half[0] - k0 : 0;
  const int lim_y = e.line < np * nx ? pa.sh.half[1] - k0 : 0;
  const int at_x = e.line * P + k0, at_y = (pl * ny + k0) * P + xx;
  const Column col{tile + (unsigned)(pl * ny + k0) * nx + xx, (unsigned)nx,
                   (unsigned)(pa.sh.half[1] * nx), lim_y};

  int64_t xa[PP], xb[PP];
  Units<PP> un;
  int key = 0;
  if constexpr (FILM) {
    // v0 = W q0 (once a segment: rows read as they lie)
    key = first_points(xa, xb, un, static_cast<const double *>(fp.in) + b * fp.in_bs, w,
                       Column{(unsigned)(e.line * nx + k0), 1u, (unsigned)pa.sh.half[0], lim_x});
  } else {
    // the units of the z lines that the points came from: the same for every plane
    const int64_t *in = static_cast<const int64_t *>(fp.in) + b * fp.in_bs + tile;
    const int16_t *u_in = fp.u_in + b * fp.u_in_bs;
    const int nt = e.ncomp, plane = ny * nx, total = np * plane;
    const int dr = nt / nx, dc = nt % nx, dp = nt % plane;
    int r = (int)threadIdx.x / nx, cc = (int)threadIdx.x % nx, ip = (int)threadIdx.x % plane;
#pragma unroll 1
    for (int i0 = threadIdx.x; i0 < total; i0 += 4 * nt) {
      int64_t x[4];
      int16_t u[4];
      int p = ip;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool on = i0 + j * nt < total;
        x[j] = on ? ld64(in + i0 + j * nt) : 0;
        u[j] = on ? __ldg(u_in + p) : (int16_t)0;
        p += dp;
        if (p >= plane) p -= plane;
      }
      ip = p;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i0 + j * nt < total) {
          S[r * P + cc] = x[j];
          us[r * P + cc] = u[j];
        }
        r += dr;
        cc += dc;
        if (cc >= nx) {
          cc -= nx;
          ++r;
        }
      }
    }
  }
  e.start();

  double *qo = static_cast<double *>(fp.q) + b * fp.q_bs;
#pragma unroll 1
  for (int f = 0; f < filters; ++f) {
    const int ax = axis_of(f);
    e.set_axis(ax);
    const int lim = ax ? lim_y : lim_x, at = ax ? at_y : at_x, st = ax ? P : 1, hs = e.H * st;
    if (FILM ? f != 0 : f != 2) {
      // a y line's points bring the units of their rows, an x line's their own, or in the
      // last filter those of their columns
      const bool own = ax == 0 && (FILM || f == 0);
      const int16_t *ur = own ? us + at : (ax ? ul + pl * ny + k0 : ul + kLines + e.line / ny * nx + k0);
      key = load_points(
          xa, xb, un, lim, [&](int i, int half) { return S[at + i * st + half * hs]; },
          [&](int i, int half) { return (int)ur[i + half * e.H]; });
    }
    key = e.line_key(f & 3, key);   // (its barrier: S is read)
    if (e.blk == 0) e.clear_key((f + 2) & 3);
    const int ue = line_unit(key);
    scale_points(xa, xb, un, ue);
    e.filter(xa, xb, []() {});
    const int uo = ue == kBadLine ? kBadUnit : ue + (ax ? shift_y : shift_x);
    const bool slice = FILM ? ax == 1 : f == 1;
    if (slice) {
      key = factor_points(xa, xb, un, w, qo, col, uo);
      if (!FILM) continue;     // v goes on along y
      if (f + 1 == filters) break;
      qo += pa.q_step;
    } else if (e.blk == 0) {
      ul[ax * kLines + e.line] = (int16_t)uo;
    }
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      if (i < lim) {
        S[at + i * st] = xa[i];
        S[at + i * st + hs] = xb[i];
        if (FILM && ax) {
          us[at + i * st] = (int16_t)un.a(i);
          us[at + i * st + hs] = (int16_t)un.b(i);
        }
      }
    }
    e.sync();
  }
  if constexpr (!FILM) {
    int64_t *out = static_cast<int64_t *>(fp.out) + b * fp.out_bs;
    over_rows(e.ncomp, nx, np * ny, [&](int r, int cc, int i) { out[tile + i] = S[r * P + cc]; });
    if (threadIdx.x < np * ny) fp.u_out[b * fp.u_out_bs + z0 * ny + threadIdx.x] = ul[threadIdx.x];
  }
  e.finish(fp.err);
}

// The same on FP32 planes (working reals between the filters).  Without a slice
// to finish (ps.qout, or a batched pass) it is the first half only: pre, x filter,
// y filter.
template <int PP>
__global__ void __launch_bounds__(544, 1)
    k_planes_f32(PlaneArgs pa, const void *tx, const void *ty, PassSet<float, kStepSet> ps) {
  typedef Tile<4, PP> E;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  E e;
  const bool half = ps.desc || !ps.qout[0];
  if (ps.desc) {
    tx = ps.desc[blockIdx.z].tc;
    ty = ps.desc[blockIdx.z].tc_y;
  }
  e.setup(smem_raw, pa.sh, tx, ty);
  const int shift_x = 23 - static_cast<const TcHead *>(tx)->kshift;
  const int shift_y = 23 - static_cast<const TcHead *>(ty)->kshift;
  const int set = set_of(ps);
  const long long b = (long long)blockIdx.z - (long long)set * ps.batch;
  const int filters = half ? 2 : 4;
  auto axis_of = [](int f) { return f == 1 || f == 2 ? 1 : 0; };
  pdl_wait();
  pdl_release();
  if (e.issuer) {
    e.run_issuer(filters, axis_of);
    e.finish(ps.err);
    return;
  }
  e.run_compute();
  const int nx = pa.nx, ny = pa.ny, P = nx + 1;
  const int z0 = blockIdx.x * pa.per, np = min(pa.per, pa.nz - z0);
  const unsigned tile = (unsigned)z0 * ny * nx;
  const int k0 = PP * e.blk, pl = e.line / nx, xx = e.line - pl * nx;
  float *S = reinterpret_cast<float *>(smem_raw);
  const float *in = ps.in[set] + b * ps.in_bs[set], *w = ps.post[set] + b * ps.w_bs;
  const float *pre = ps.pre[set] ? ps.pre[set] + b * ps.w_bs : nullptr;
  float *out = ps.out[set] + b * ps.out_bs[set], *qo = ps.qout[set] + b * ps.qout_bs[set];
  if (ps.desc) {
    const PassDesc d = ps.desc[blockIdx.z];
    in = d.in;
    out = d.out;
    pre = d.pre;
  }
  const int lim_x = e.line < np * ny ? pa.sh.half[0] - k0 : 0;
  const int lim_y = e.line < np * nx ? pa.sh.half[1] - k0 : 0;
  const int at_x = e.line * P + k0, at_y = (pl * ny + k0) * P + xx;
  const unsigned off = tile + (unsigned)(pl * ny + k0) * nx + xx, ghs = pa.sh.half[1] * nx;
  if (pre)
    over_rows<8>(e.ncomp, nx, np * ny,
                 [&](int i) { return WithFactor<float>{__ldg(in + tile + i), __ldg(pre + tile + i)}; },
                 [&](int r, int cc, int, WithFactor<float> v) { S[r * P + cc] = v.x * v.w; });
  else
    over_rows<8>(e.ncomp, nx, np * ny, [&](int i) { return __ldg(in + tile + i); },
                 [&](int r, int cc, int, float x) { S[r * P + cc] = x; });
  e.start();
#pragma unroll 1
  for (int f = 0; f < filters; ++f) {
    const int ax = axis_of(f);
    e.set_axis(ax);
    const int lim = ax ? lim_y : lim_x, at = ax ? at_y : at_x, st = ax ? P : 1, hs = e.H * st;
    float ya[PP], yb[PP];
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      ya[i] = i < lim ? S[at + i * st] : 0.f;
      yb[i] = i < lim ? S[at + i * st + hs] : 0.f;
    }
    int key = 0;
#pragma unroll
    for (int i = 0; i < PP; ++i) key = max(key, max(mag_key(ya[i]), mag_key(yb[i])));
    key = e.line_key(f, key);   // (its barrier: S is read)
    const bool bad = key >= bad_key<float>();
    const int Eb = line_exp(0.f, key), ue = unit_exp(0.f, Eb) + (ax ? shift_y : shift_x);
    int xa[PP], xb[PP];
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      xa[i] = to_fixed(ya[i], Eb);
      xb[i] = to_fixed(yb[i], Eb);
    }
    e.filter(xa, xb, []() {}, [&](int i, float p, float q) {
      ya[i] = bad ? bad_value(0.f) : scale2(p, ue);
      yb[i] = bad ? bad_value(0.f) : scale2(q, ue);
    });
    if (f == 1 && !half) {
#pragma unroll
      for (int g = 0; g < PP; g += 4) {
        float w0[4], w1[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          w0[i] = g + i < lim ? __ldg(w + (off + (g + i) * nx)) : 0.f;
          w1[i] = g + i < lim ? __ldg(w + (off + (g + i) * nx + ghs)) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float q0 = ya[g + i] * w0[i], q1 = yb[g + i] * w1[i];
          if (g + i < lim) {
            qo[off + (g + i) * nx] = q0;
            qo[off + (g + i) * nx + ghs] = q1;
          }
          ya[g + i] = q0 * w0[i];
          yb[g + i] = q1 * w1[i];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      if (i < lim) {
        S[at + i * st] = ya[i];
        S[at + i * st + hs] = yb[i];
      }
    }
    e.sync();
  }
  over_rows(e.ncomp, nx, np * ny, [&](int r, int cc, int i) { out[tile + i] = S[r * P + cc]; });
  e.finish(ps.err);
}

// Geometry of a pass, or false when the kernels do not take it.
bool lines_of(const AxisPlan &ap, int nd, Lines &ln) {
  if (!ap.tc || !tc_line_possible(ap.n, nd) || ap.n_real < 1 || ap.n_outer < 1) return false;
  const int kg = line_blocks(ap.n);
  memset(&ln.sh, 0, sizeof ln.sh);
  ln.sh.nd = nd;
  ln.sh.pp = pairs_per_thread(kg);
  ln.sh.rep = 1;
  ln.sh.axes = 1;
  ln.sh.half[0] = ln.sh.half[1] = ap.n / 2;
  ln.sh.kg[0] = ln.sh.kg[1] = kg;
  ln.n = ap.n;
  ln.s_n = ap.s_n;
  ln.lines = (long long)ap.n_real * ap.n_outer;
  if (ap.n_fast) {                 // rows
    ln.row_len = 1;
    ln.s_outer = ap.n;
  } else if (ap.flat_nx) {         // columns over (row, outer)
    ln.row_len = ap.flat_nx;
    ln.s_outer = ap.s_outer;
  } else {
    ln.row_len = ap.n_real;
    ln.s_outer = ap.s_outer;
  }
  return (ln.lines + kLines - 1) / kLines <= 0x7fffffffLL;
}

// Copies of each line per CTA, and with them 4 points per thread, so that small
// launches of lines of up to 64 points spread over the SMs: doubled while both
// chains' CTAs still fit there side by side (ms per SCF iteration, one copy
// against this: FP64 16^3 3.34 / 2.05, 32^3 3.87 / 2.24, 64^3 5.57 / 3.88, 64 x 64 x 1 3.37 /
// 2.18).  With 16 points per thread two copies were slower (FP32 100 x 80 x 60 5.7 against
// 5.2).
void spread(Shape &sh, long long lines) {
  if (sh.pp == 16) return;
  const int kg = sh.axes == 2 ? std::max(sh.kg[0], sh.kg[1]) : sh.kg[0];
  while (sh.rep < 4 && 2 * ((lines + kLines / (2 * sh.rep) - 1) / (kLines / (2 * sh.rep))) <= 152 &&
         16 * kg >= 8 * sh.rep)
    sh.rep *= 2;
  if (sh.rep > 1 && sh.pp == 8) sh.pp = 4;
}
inline int lines_per_cta(const Shape &sh) { return kLines / sh.rep; }

template <typename T, int MAXT, int PP, bool XP, bool PR>
cudaError_t launch_real_t(Lines ln, const void *tc, const PassSet<T, kStepSet> &ps, cudaStream_t st) {
  const int lc = lines_per_cta(ln.sh);
  dim3 grid((unsigned)((ln.lines + lc - 1) / lc), 1, ps.nset * ps.batch);
  ln.sh.stage = XP ? lc * (ln.n + 1) * (int)sizeof(T) : 0;
  ln.sh.finish();
  return launch_pdl(k_real<T, MAXT, PP, XP, PR>, grid, dim3(ln.sh.threads),
                    (size_t)ln.sh.lay.total, st, ln, tc, ps);
}
template <typename T, bool XP, bool PR>
cudaError_t launch_real_kg(Lines ln, const void *tc, const PassSet<T, kStepSet> &ps, cudaStream_t st) {
  spread(ln.sh, ln.lines * ps.nset * ps.batch);
  if (ln.sh.pp == 4) return launch_real_t<T, 544, 4, XP, PR>(ln, tc, ps, st);
  if (ln.sh.pp == 8) return launch_real_t<T, 544, 8, XP, PR>(ln, tc, ps, st);
  if constexpr (std::is_same<T, float>::value) {
    if (ln.sh.kg[0] > 4) return launch_real_t<T, 1024, 16, XP, PR>(ln, tc, ps, st);
  }
  return launch_real_t<T, 640, 16, XP, PR>(ln, tc, ps, st);
}
template <typename T>
cudaError_t launch_real(const AxisPlan &ap, const PassSet<T, kStepSet> &ps, bool pair, cudaStream_t st) {
  Lines ln;
  const long long sets = (long long)ps.nset * ps.batch;
  if (!lines_of(ap, kNd<T>, ln) || ps.nset < 1 || ps.nset > kStepSet || sets < 1 || sets > 65535 ||
      (ps.desc && (pair || kNd<T> != 4)))
    return cudaErrorInvalidValue;
  for (int k = 0; k < ps.nset && !ps.desc; ++k) {
    if (!ps.in[k] || !ps.out[k] || (pair && (!ps.post[k] || !ps.qout[k])))
      return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(ps.in[k]) | reinterpret_cast<uintptr_t>(ps.out[k]) |
         reinterpret_cast<uintptr_t>(ps.pre[k]) | reinterpret_cast<uintptr_t>(ps.post[k]) |
         reinterpret_cast<uintptr_t>(ps.qout[k])) & (sizeof(T) - 1))
      return cudaErrorMisalignedAddress;
  }
  if constexpr (std::is_same<T, float>::value) {
    if (pair)
      return ap.n_fast ? launch_real_kg<T, true, true>(ln, ap.tc, ps, st)
                       : launch_real_kg<T, false, true>(ln, ap.tc, ps, st);
  } else {
    if (pair) return cudaErrorInvalidValue;   // 64-bit pairs run in k_fix
  }
  return ap.n_fast ? launch_real_kg<T, true, false>(ln, ap.tc, ps, st)
                   : launch_real_kg<T, false, false>(ln, ap.tc, ps, st);
}

template <bool XP, int MODE>
cudaError_t launch_fix_t(Lines ln, const void *tc, const FixPass &fp, cudaStream_t st) {
  spread(ln.sh, ln.lines * fp.batch);
  const int lc = lines_per_cta(ln.sh);
  dim3 grid((unsigned)((ln.lines + lc - 1) / lc), 1, fp.batch);
  // x passes stage rows; column passes with 16 points per thread the factor step
  // (and 2 bytes for each point's unit)
  if (XP) {
    ln.sh.stage = lc * (ln.n + 1) * 8;
    ln.sh.units = lc * (ln.n + 1) * 2;
  } else if (ln.sh.pp == 16) {
    if (MODE == PAIR || MODE == LAST) {
      ln.sh.stage = kLines * ln.sh.kg[0] * 256;
      ln.sh.units = kLines * ln.sh.kg[0] * 64;
    }
  }
  ln.sh.finish();
  const size_t smem = ln.sh.lay.total;
  if (ln.sh.pp == 4)
    return launch_pdl(k_fix<4, XP, MODE>, grid, dim3(ln.sh.threads), smem, st, ln, tc, fp);
  if (ln.sh.pp == 8)
    return launch_pdl(k_fix<8, XP, MODE>, grid, dim3(ln.sh.threads), smem, st, ln, tc, fp);
  return launch_pdl(k_fix<16, XP, MODE>, grid, dim3(ln.sh.threads), smem, st, ln, tc, fp);
}

// Planes of nx x ny points, nz of them per instance (film: a march segment).
void plane_shape(int nx, int ny, int nz, int nd, int batch, bool film, PlaneArgs &pa) {
  memset(&pa, 0, sizeof pa);
  pa.nx = nx;
  pa.ny = ny;
  pa.nz = nz;
  pa.sh.nd = nd;
  pa.sh.pp = 8;
  pa.sh.rep = 1;
  pa.sh.axes = 2;
  pa.sh.half[0] = nx / 2;
  pa.sh.half[1] = ny / 2;
  pa.sh.kg[0] = line_blocks(nx);
  pa.sh.kg[1] = line_blocks(ny);
  const int m = std::max(nx, ny), per = kLines / m;
  // a film's one plane: as many copies of its lines as fit; else by the lines
  // that the planes fill if a CTA takes 128 of them
  spread(pa.sh, film ? 1 : (long long)((nz + per - 1) / per) * kLines * batch);
  while (lines_per_cta(pa.sh) < m) pa.sh.rep /= 2;
  pa.sh.pp = pa.sh.rep > 1 ? 4 : 8;
  const int lc = lines_per_cta(pa.sh);
  pa.per = lc / m;
  pa.sh.stage = lc * (nx + 1) * (nd == 7 ? 8 : 4);
  pa.sh.units = nd == 7 ? lc * (nx + 1) * 2 : 0;
  pa.sh.finish();
}
// ... of passes apx (x) and apy (lines nx apart), or false.
bool planes_of(const AxisPlan &apx, const AxisPlan &apy, int nd, int batch, bool film,
               PlaneArgs &pa) {
  Lines lx, ly;
  if (!lines_of(apx, nd, lx) || !lines_of(apy, nd, ly) || !apx.n_fast || apy.n_fast ||
      apy.s_n != apx.n || lx.sh.pp > 8 || ly.sh.pp > 8)
    return false;
  plane_shape(apx.n, apy.n, (int)(lx.lines / apy.n), nd, batch, film, pa);
  return true;
}

// Shared-memory opt-in; *fits goes false where the compiler's register count of a
// kernel that splits them does not hold the split.
template <typename K> cudaError_t opt_in(K *k, bool *fits = nullptr) {
  if (fits) {
    cudaFuncAttributes at;
    const cudaError_t e = cudaFuncGetAttributes(&at, k);
    if (e != cudaSuccess) return e;
    for (int c = 2; c <= 4; ++c) *fits = *fits && split_fits(at.numRegs, c);
  }
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}
template <typename T, int MAXT, int PP> cudaError_t prep_real(bool *split) {
  bool *fits = kNd<T> == 7 && PP == 16 ? split : nullptr;
  cudaError_t e;
  if ((e = opt_in(k_real<T, MAXT, PP, true, false>, fits)) != cudaSuccess) return e;
  if ((e = opt_in(k_real<T, MAXT, PP, false, false>, fits)) != cudaSuccess) return e;
  if constexpr (std::is_same<T, float>::value) {
    if ((e = opt_in(k_real<T, MAXT, PP, true, true>, fits)) != cudaSuccess) return e;
    if ((e = opt_in(k_real<T, MAXT, PP, false, true>, fits)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}
template <int PP> cudaError_t prep_fix(bool *split) {
  bool *fits = PP == 16 ? split : nullptr;
  cudaError_t e;
  if constexpr (PP <= 8) {
    if ((e = opt_in(k_planes<PP, false>)) != cudaSuccess) return e;
    if ((e = opt_in(k_planes<PP, true>)) != cudaSuccess) return e;
    if ((e = opt_in(k_planes_f32<PP>)) != cudaSuccess) return e;
  }
  if ((e = opt_in(k_fix<PP, true, FIRST>, fits)) != cudaSuccess) return e;
  if ((e = opt_in(k_fix<PP, false, FIRST>, fits)) != cudaSuccess) return e;
  if ((e = opt_in(k_fix<PP, false, MID>, fits)) != cudaSuccess) return e;
  if ((e = opt_in(k_fix<PP, true, PAIR>, fits)) != cudaSuccess) return e;
  if ((e = opt_in(k_fix<PP, false, PAIR>, fits)) != cudaSuccess) return e;
  if ((e = opt_in(k_fix<PP, true, LAST>, fits)) != cudaSuccess) return e;
  return opt_in(k_fix<PP, false, LAST>, fits);
}

// ---- host: the convolution kernel in double-double arithmetic
struct dd {
  double h, l;
};
dd dd_norm(double a, double b) {
  const double s = a + b, bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
dd dd_add(dd a, dd b) {
  dd s = dd_norm(a.h, b.h);
  return dd_norm(s.h, s.l + (a.l + b.l));
}
dd dd_mul(dd a, dd b) {
  const double p = a.h * b.h, e = fma(a.h, b.h, -p);
  return dd_norm(p, e + (a.h * b.l + a.l * b.h));
}
dd dd_div_small(dd a, double n) {   // a / n, n a small integer
  const double q = a.h / n, r = fma(-q, n, a.h);
  return dd_norm(q, (r + a.l) / n);
}
// cos(2 pi m / n): Taylor series on [0, pi/4], the symmetries outside
dd dd_cos2pi(long m, long n) {
  m %= n;
  if (2 * m > n) m = n - m;                 // cos is even: m/n in [0, 1/2]
  bool neg = false;
  if (4 * m > n) {                          // cos(pi - t) = -cos t
    m = n - 2 * m;
    n *= 2;
    neg = true;
  }
  const bool sine = 8 * m > n;              // above 1/8: cos(pi/2 - t) = sin t
  if (sine) {
    m = n - 4 * m;
    n *= 4;
  }
  const dd two_pi = {6.283185307179586, 2.4492935982947064e-16};
  dd x = dd_mul(two_pi, dd_div_small({(double)m, 0.0}, (double)n));
  dd x2 = dd_mul(x, x), term = sine ? x : dd{1.0, 0.0}, sum = term;
  for (int i = 1; i < 20; ++i) {
    const double d = sine ? (2.0 * i) * (2.0 * i + 1.0) : (2.0 * i - 1.0) * (2.0 * i);
    term = dd_div_small(dd_mul(term, x2), -d);
    sum = dd_add(sum, term);
    if (fabs(term.h) < 1e-36) break;
  }
  return neg ? dd{-sum.h, -sum.l} : sum;
}
// a * 2^s as an integer, rounded to nearest (|a 2^s| < 2^62)
int64_t dd_to_int(dd a, int s) {
  const double h = ldexp(a.h, s), l = ldexp(a.l, s);
  const double hi = rint(h);
  const double r = rint((h - hi) + l);
  return (int64_t)hi + (int64_t)r;
}
// a small integer as f16 bits
uint16_t f16_of_int(int v) {
  if (v == 0) return 0;
  const uint16_t s = v < 0 ? 0x8000 : 0;
  int a = v < 0 ? -v : v, e = 0;
  while ((a >> (e + 1)) != 0) ++e;
  return (uint16_t)(s | ((15 + e) << 10) | (((a << (10 - e)) & 0x3ff)));
}
// digit j (0 the top one) of v
int digit_of(int64_t v, int nd, int j) {
  const uint64_t z = (uint64_t)v + (nd == 7 ? 0x0080808080808080ULL : 0x80808080ULL);
  return (int)((z >> (8 * (nd - 1 - j))) & 0xff) - 128;
}

// The table with K scaled `less` bits below the digits' full range.
bool build_scaled(const std::vector<dd> &K, int nd, int kg, int less,
                  std::vector<unsigned char> &table) {
  const int n = (int)K.size(), H = n / 2, kp = 16 * kg;
  const int bits = 8 * nd;
  double mx = 0.0, l1 = 0.0;
  for (int d = 0; d < H; ++d) {
    for (int s = -1; s <= 1; s += 2) mx = fmax(mx, fabs(K[d].h + s * K[d + H].h));
    l1 += fabs(K[d].h) + fabs(K[d + H].h);
  }
  TcHead head;
  memset(&head, 0, sizeof head);
  int shift = 0;
  if (mx > 0.0) {
    int ex;
    frexp(mx, &ex);                               // mx < 2^ex
    shift = bits - 1 - ex;
    // a top digit of at most 127 with any others behind it
    if (ldexp(mx, shift) > ldexp(126.9, bits - 8)) --shift;
    // results |2 y| <= sum |K'| * 2^(kFine - 1) below 2^61
    while (nd == 7 && ldexp(l1, shift) > 0x1.fp61 / (1 << kFine)) --shift;
  }
  shift -= less;
  if (shift > 900 || shift < -900) return false;
  head.kshift = shift;
  // integers of K, with the zero-frequency sum kept exact: its rounding would
  // act on every line's mean in every step
  std::vector<int64_t> Ki(n);
  dd sum = {0.0, 0.0};
  int64_t isum = 0;
  for (int d = 0; d < n; ++d) {
    Ki[d] = dd_to_int(K[d], shift);
    isum += Ki[d];
    sum = dd_add(sum, K[d]);
  }
  int64_t miss = dd_to_int(sum, shift) - isum;
  for (int d = 1; (miss > 1 || miss < -1) && 2 * d < n; ++d) {   // in +-d pairs near the peak
    const int s = miss > 0 ? 1 : -1;
    Ki[d] += s;
    Ki[n - d] += s;
    miss -= 2 * s;
  }
  Ki[0] += miss;
  table.assign(tc_table_bytes(n, nd), 0);
  uint16_t *out = reinterpret_cast<uint16_t *>(table.data() + sizeof(TcHead));
  for (int par = 0; par < 2; ++par) {
    // t[d], d = n - k in (-H, H): cyclic (c) or negacyclic (d)
    auto tv = [&](int d) -> int64_t {
      if (d <= -H || d >= H) return 0;
      const int m = d < 0 ? d + H : d;
      const int64_t v = par == 0 ? Ki[m] + Ki[m + H] : Ki[m] - Ki[m + H];
      return par == 1 && d < 0 ? -v : v;
    };
    double worst = 0.0;
    for (int d = 0; d < H; ++d) {
      const int64_t v = tv(d);
      // for d also -v can stand in a row: the larger digit bounds the sums
      for (int j = 0; j < nd; ++j) {
        const int a = abs(digit_of(v, nd, j)), c = par == 1 ? abs(digit_of(-v, nd, j)) : 0;
        worst += 128.0 * std::max(a, c);
      }
    }
    if (!(worst < (nd == 7 ? 4194304.0 : 16777216.0))) return false;
    uint16_t *half = out + (size_t)par * b_half_bytes(nd, kg) / 2;
    // digits by offset, then the blocks by look-up (each offset stands in up to 64
    // rows: 64 points 240 us -> 50 us a table)
    const int far = kp + 8;                  // offsets -far .. far, 0 outside the line
    std::vector<uint16_t> dig((size_t)nd * (2 * far + 1), 0);
    for (int d = 1 - H; d < H; ++d)
      for (int j = 0; j < nd; ++j)
        dig[(size_t)j * (2 * far + 1) + far + d] = f16_of_int(digit_of(tv(d), nd, j));
    auto row_of = [&](int j, int d) { return &dig[(size_t)j * (2 * far + 1) + far + d]; };
    if (dense_b(kg)) {       // [k block][row block of (round, digit, output)][8 rows][8 k]
      const int rounds = split_rows(nd, kg) ? 2 : 1, gc = group_cols(nd, kg);
      for (int rd = 0; rd < rounds; ++rd)
        for (int j = 0; j < nd; ++j)
          for (int col = 0; col < gc; ++col) {
            const int r = rounds == 2 ? col / 8 * 16 + 8 * rd + col % 8 : col;   // the output
            if (r >= H) continue;
            const int row = (rd * nd + j) * gc + col;
            const uint16_t *t = row_of(j, r);
            for (int k0 = 0; k0 < H; k0 += 8) {
              uint16_t *o = half + ((size_t)(k0 / 8) * (rounds * nd * gc / 8) + row / 8) * 64 + (row % 8) * 8;
              for (int k = k0; k < k0 + 8 && k < H; ++k) o[k - k0] = t[-k];
            }
          }
    } else {                 // [digit][n block - k block][8][8]
      const int NB = 4 * kg - 1;
      for (int j = 0; j < nd; ++j)
        for (int blk = 0; blk < NB; ++blk)
          for (int r = 0; r < 8; ++r)
            for (int c = 0; c < 8; ++c)
              half[((size_t)j * NB + blk) * 64 + r * 8 + c] = *row_of(j, 8 * (blk - (2 * kg - 1)) + r - c);
    }
  }
  memcpy(table.data(), &head, sizeof head);
  return true;
}

}  // namespace

bool tc_line_possible(int n, int nd) {
  return n >= 2 && n % 2 == 0 && line_blocks(n) <= (nd == 4 ? 7 : 4);
}

size_t tc_table_bytes(int n, int nd) {
  const int kg = line_blocks(n);
  return sizeof(TcHead) + 2 * (size_t)b_half_bytes(nd, kg);
}

// CTAs of a pass of one instance.
long long tc_pass_ctas(const AxisPlan &ap, int nd) {
  Lines ln;
  if (!lines_of(ap, nd, ln)) return 0;
  spread(ln.sh, ln.lines);
  const int lc = lines_per_cta(ln.sh);
  return (ln.lines + lc - 1) / lc;
}

// Whether a step's x and y passes run on whole planes.  A film's do when a
// segment can stay in one CTA's 128 threads' reach, that is at up to 32 x 32
// (ms per SCF iteration with 200 steps, planes against passes: 32 x 32 1.32 / 1.69,
// 500 of them 5.0 / 9.1; with one unit per instance 40 x 36 1.95 / 1.84, 64 x 64 2.01 /
// 1.94).  Otherwise
// planes save two launches in two steps, but a plane does not split over CTAs,
// its lines leave part of the 128 rows idle, and its CTAs may need one wave
// more.  The filters' time on both sides is taken as the waves of both chains'
// CTAs times 2 + 4/rep; in that unit (0.6 us for 7 digits, 0.35 us for 4) a launch
// saved is worth 2 and 4.  Measured: for planes FP64 32^3 2.17 / 2.54, 56^3 3.81 / 4.05,
// 64^3 3.81 / 4.22 and FP32 60^3 2.13 / 2.50, 36^3 1.81 / 2.05; against them FP64 48^3 3.47 /
// 3.38, 40^3 3.30 / 3.27, and with one unit per instance (12, 20, 28) x 8 2.63 / 2.31,
// (64, 40, 30) x 4 4.55 / 4.23, (36, 36, 38) x 20 14.2 / 12.9 and FP32 8.8 / 8.6.
bool tc_planes_wanted(int nx, int ny, int nz, int nd, int batch) {
  if (nx > kLines / 2 || ny > kLines / 2 || nx < 2 || ny < 2) return false;
  if (nz == 1) return nx <= 32 && ny <= 32;
  auto cost = [&](long long ctas, int rep) {
    return (double)((2 * ctas + 151) / 152) * (2.0 + 4.0 / rep);
  };
  auto pass = [&](int n, long long lines) {
    Shape sh = {};
    sh.nd = nd;
    sh.pp = 8;
    sh.rep = sh.axes = 1;
    sh.kg[0] = line_blocks(n);
    spread(sh, lines * batch);
    const int lc = lines_per_cta(sh);
    return cost((lines + lc - 1) / lc * batch, sh.rep);
  };
  PlaneArgs pa;
  plane_shape(nx, ny, nz, nd, batch, false, pa);
  const double planes = 2.0 * cost((long long)((nz + pa.per - 1) / pa.per) * batch, pa.sh.rep);
  return planes < pass(nx, (long long)ny * nz) + pass(ny, (long long)nx * nz) + (nd == 7 ? 2.0 : 4.0);
}

// Digits of the two half-length kernels of gain table g (natural order, real
// and even, the 1/n of the transform included).  The digits' sizes depend on
// the scale; the first of a few scales whose accumulators stay in the exact
// range is taken.  False when none does or the gains are not finite: the
// caller keeps the FFT pass.  row_sum: sum |K|, the filter's largest growth.
bool tc_build_table(const double *g, int n, int nd, std::vector<unsigned char> &table,
                    double *row_sum) {
  for (int k = 0; k < n; ++k)
    if (!std::isfinite(g[k])) return false;
  std::vector<dd> ct(n), K(n);
  for (int m = 0; 2 * m <= n; ++m) ct[m] = ct[(n - m) % n] = dd_cos2pi(m, n);
  double l1 = 0.0;
  // g and K are even: bins and offsets up to n/2 stand for their mirrors
  const int h = n / 2;
  for (int d = 0; d <= h; ++d) {
    dd s = {0.0, 0.0};
    for (int k = 1; k < h; ++k) s = dd_add(s, dd_mul({g[k], 0.0}, ct[k * d % n]));
    s = dd_add({2.0 * s.h, 2.0 * s.l}, {g[0], 0.0});
    K[d] = dd_add(s, {d & 1 ? -g[h] : g[h], 0.0});
    if (d > 0 && d < h) K[n - d] = K[d];
    l1 += fabs(K[d].h) * (d > 0 && d < h ? 2.0 : 1.0);
  }
  if (row_sum) *row_sum = l1;
  for (int less = 0; less < 4; ++less)
    if (build_scaled(K, nd, line_blocks(n), less, table)) return true;
  return false;
}

namespace {
cudaError_t prepare_all(bool *split) {
  cudaError_t e;
  if ((e = prep_real<float, 544, 4>(split)) != cudaSuccess) return e;
  if ((e = prep_real<double, 544, 4>(split)) != cudaSuccess) return e;
  if ((e = prep_fix<4>(split)) != cudaSuccess) return e;
  if ((e = prep_real<float, 544, 8>(split)) != cudaSuccess) return e;
  if ((e = prep_real<float, 640, 16>(split)) != cudaSuccess) return e;
  if ((e = prep_real<float, 1024, 16>(split)) != cudaSuccess) return e;
  if ((e = prep_real<double, 544, 8>(split)) != cudaSuccess) return e;
  if ((e = prep_real<double, 640, 16>(split)) != cudaSuccess) return e;
  if ((e = prep_fix<8>(split)) != cudaSuccess) return e;
  return prep_fix<16>(split);
}
struct Prepared {
  std::mutex mu;
  bool done[64] = {}, split[64] = {};
};
Prepared &prepared() {
  static Prepared p;
  return p;
}
}  // namespace

// Kernel attributes, set once per device (host threads may race to it).
cudaError_t tc_prepare() {
  Prepared &p = prepared();
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(p.mu);
  if (!p.done[dev]) {
    p.split[dev] = true;
    if ((e = prepare_all(&p.split[dev])) != cudaSuccess) return e;
    p.done[dev] = true;
  }
  return cudaSuccess;
}
// Whether the kernels of such lines can run on the current device (prepared):
// without the register split 64-bit lines above 64 points keep their FFT passes.
bool tc_line_usable(int n, int nd) {
  if (!tc_line_possible(n, nd)) return false;
  Prepared &p = prepared();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  std::lock_guard<std::mutex> lock(p.mu);
  return p.done[dev] && (p.split[dev] || !split_rows(nd, line_blocks(n)));
}

cudaError_t launch_tc(const AxisPlan &ap, const PassSet<float, kStepSet> &ps, bool pair, cudaStream_t st) {
  return launch_real(ap, ps, pair, st);
}
cudaError_t launch_tc(const AxisPlan &ap, const PassSet<double, kStepSet> &ps, bool pair, cudaStream_t st) {
  return launch_real(ap, ps, pair, st);
}

cudaError_t launch_fix(const AxisPlan &ap, int mode, const FixPass &fp, cudaStream_t st) {
  Lines ln;
  if (!lines_of(ap, 7, ln) || fp.batch < 1 || fp.batch > 65535 || !fp.in ||
      (mode != LAST && (!fp.out || !fp.u_out)) || (mode != FIRST && (!fp.u_in || fp.u_div < 1)) ||
      (mode != MID && !fp.w) || ((mode == PAIR || mode == LAST) && !fp.q))
    return cudaErrorInvalidValue;
  const bool x = ap.n_fast != 0;
  switch (mode) {
    case FIRST:
      return x ? launch_fix_t<true, FIRST>(ln, ap.tc, fp, st)
               : launch_fix_t<false, FIRST>(ln, ap.tc, fp, st);
    case MID:
      return x ? cudaErrorInvalidValue : launch_fix_t<false, MID>(ln, ap.tc, fp, st);
    case PAIR:
      return x ? launch_fix_t<true, PAIR>(ln, ap.tc, fp, st)
               : launch_fix_t<false, PAIR>(ln, ap.tc, fp, st);
    case LAST:
      return x ? launch_fix_t<true, LAST>(ln, ap.tc, fp, st)
               : launch_fix_t<false, LAST>(ln, ap.tc, fp, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_planes(const AxisPlan &apx, const AxisPlan &apy, const PassSet<float, kStepSet> &ps,
                          cudaStream_t st) {
  PlaneArgs pa;
  const long long sets = (long long)ps.nset * ps.batch;
  if (ps.nset < 1 || ps.nset > kStepSet || sets < 1 || sets > 65535 ||
      !planes_of(apx, apy, 4, (int)sets, false, pa))
    return cudaErrorInvalidValue;
  for (int k = 0; k < ps.nset && !ps.desc; ++k)
    if (!ps.in[k] || !ps.out[k] || !ps.qout[k] != !ps.qout[0] || (ps.qout[0] && !ps.post[k]) ||
        (ps.qout[0] && ps.pre[k]) || (!ps.qout[0] && ps.post[k]))
      return cudaErrorInvalidValue;
  dim3 grid((pa.nz + pa.per - 1) / pa.per, 1, (unsigned)sets);
  const size_t smem = pa.sh.lay.total;
  return launch_pdl(pa.sh.pp == 4 ? k_planes_f32<4> : k_planes_f32<8>, grid, dim3(pa.sh.threads),
                    smem, st, pa, apx.tc, apy.tc, ps);
}
// steps 0: the fused step on planes; else a film's segment of that many steps
// (fp.q: the first finished slice, q_step to the next one).
cudaError_t launch_planes(const AxisPlan &apx, const AxisPlan &apy, const FixPass &fp, int steps,
                          long long q_step, cudaStream_t st) {
  PlaneArgs pa;
  if (!planes_of(apx, apy, 7, fp.batch, steps > 0, pa) || fp.batch < 1 || fp.batch > 65535 || !fp.in ||
      !fp.w || !fp.q || (steps == 0 && (!fp.u_in || !fp.u_out || !fp.out)) || steps < 0 ||
      (steps > 0 && pa.nz != 1))
    return cudaErrorInvalidValue;
  pa.steps = steps;
  pa.q_step = q_step;
  dim3 grid((pa.nz + pa.per - 1) / pa.per, 1, fp.batch);
  const size_t smem = pa.sh.lay.total;
  auto k = steps ? (pa.sh.pp == 4 ? k_planes<4, true> : k_planes<8, true>)
                 : (pa.sh.pp == 4 ? k_planes<4, false> : k_planes<8, false>);
  return launch_pdl(k, grid, dim3(pa.sh.threads), smem, st, pa, apx.tc, apy.tc, fp);
}

}  // namespace scft
