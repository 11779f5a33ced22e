// Core of the tensor-core line filters (k_tc.cu): one axis of the separable
// split-step operator as an exact integer convolution.
//
// The pass IFFT . diag(g) . FFT along an axis of N points is the circulant
// convolution y[n] = sum_k K[(n-k) mod N] x[k] with K = IDFT(g).  Splitting it
// by z^N - 1 = (z^H - 1)(z^H + 1), H = N/2, leaves two H x H Toeplitz products
//   c = Kc (x[k] + x[k+H]),  d = Kd (x[k] - x[k+H]),   Kc/Kd = K[d] +- K[d+H]
//   y[n] = (c[n] + d[n])/2,  y[n+H] = (c[n] - d[n])/2 .
// Each is computed without rounding (the slicing scheme of Ozaki, Ogita, Oishi
// and Rump, Numer. Algorithms 59, 2012): the line and the kernel are integers
// of ND base-256 digits (slices.cuh; FP64 7, FP32 4), a digit
// is an exact f16 number, and the products of digits i and j with i + j = g
// accumulate in FP32 in one TMEM accumulator per g.  The host checks for each
// table that no accumulator can reach 2^22 (2^24 for FP32), so every partial
// sum is an integer that FP32 holds exactly and the order of the sums does not
// matter.  What is left out (i + j >= ND, for 7 digits i + j >= 8: groups 0 .. 7 are kept)
// is below the last digit's unit.  The eighth group and an output unit 4 bits finer
// (kFine) leave less at the small values of a line than an FFT does: with
// seven groups and the coarser unit values 2^-90 of a line's largest were up to 5 times
// further off.
//
// Tile: the 128 rows (M) of one tcgen05.mma x N points per CTA.  A row holds one
// of LN = 128/rep lines; with rep > 1 every line stands in rep rows, because a
// thread reaches only its own TMEM lane: the threads of a line's copies share
// its points out, so that a small grid spreads over rep times as many CTAs.
// Thread t owns row t % 128 and the PP points k = PP*blk + i with their partners
// k + H: it writes their digits as A operands, once per copy (K-major core
// matrices of 8 rows x 16 bytes, unswizzled), and reads the same outputs back.
// B holds the digits of Kc or Kd stacked along its rows (digit j, output n), so
// one instruction multiplies x's digit i with all of K's digits that it meets (the
// first ND-i; 7 digits: 8-i, at most 7) and adds into the accumulators from i on side
// by side: up to 256 columns per instruction.  (One instruction per digit pair, 32 or 64 columns wide, took
// about 76 cycles each whatever its width.)  Lines above 128 points (FP32) have
// no room for that B; there its 8x8 core matrix (bn, bk), which depends only on
// bn - bk, is shared by descriptor: with A's k blocks in reverse order both
// strides are one core matrix.
#pragma once

#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "slices.cuh"

namespace scft {
namespace tc {

using namespace slices;

constexpr int kLines = 128;

// Scales of a table, in front of its digits (device memory: a box change
// rewrites tables in place under captured graphs).
struct TcHead {
  int kshift;    // K' = K * 2^kshift
  int pad[3];
};
// 7 digits: bits of a result below 256^7, the unit of K' X / 256^6 / 256.  Its 61 bits
// bound K': sum |K'| < 2^(62 - kFine).
constexpr int kFine = 4;
// accumulators (digit groups) of a product
__host__ __device__ constexpr int groups(int nd) { return nd == 7 ? 8 : nd; }

// 16-point blocks of a half line
__host__ __device__ constexpr int line_blocks(int n) { return (n / 2 + 15) / 16; }
// Points per thread: 16 on lines above 64 points (512 computing threads at 128),
// else 8, or 4 in CTAs of fewer lines.
__host__ __device__ constexpr int pairs_per_thread(int kg) { return kg <= 2 ? 8 : 16; }
__host__ __device__ constexpr bool dense_b(int kg) { return kg <= 4; }
// Accumulators come in two TMEM buffers, so that one is read while the tensor
// core fills the other.  A buffer holds all outputs of c or d (whose A operands
// then lie side by side); for 7 digits (8 accumulators) and 16 points per thread TMEM and shared
// memory have no room for that: a buffer holds half of the outputs (8 of each
// thread's 16), a half takes two rounds, and c's operand memory serves d.
__host__ __device__ constexpr bool split_rows(int nd, int kg) { return nd == 7 && kg > 2; }
__host__ __device__ constexpr bool both_halves(int nd, int kg) {
  return !split_rows(nd, kg) && dense_b(kg);
}
// Accumulator columns of one digit group in one buffer (a multiple of 16).
__host__ __device__ constexpr int group_cols(int nd, int kg) {
  return split_rows(nd, kg) ? 32 : 16 * kg;
}
__host__ __device__ constexpr int b_half_bytes(int nd, int kg) {
  return dense_b(kg) ? nd * group_cols(nd, kg) * (split_rows(nd, kg) ? 2 : 1) * (16 * kg) * 2
                     : nd * (4 * kg - 1) * 128;
}
// The issuing warp; with 16 points per thread and 7 digits a warpgroup of its
// own, so that the computing ones can take its registers (setmaxnreg).  112 + 24
// left the issuing warp too few: it kept its loop in local memory.
__host__ __device__ constexpr int issuer_threads(int pp) { return pp == 16 ? 128 : 32; }
constexpr int kRegsCompute = 104, kRegsIssue = 56;
// Whether a block of 128 c computing threads and the issuing 128, launched with
// `regs` registers a thread, holds what the split asks for (the computing threads
// would wait for ever otherwise): 96 do for every c (104 x 512 + 56 x 128 = 60416 <= 96 x
// 640 = 61440; 47104 <= 49152 for 3, 33792 <= 36864 for 2).
__host__ __device__ constexpr bool split_fits(int regs, int c) {
  return regs >= kRegsIssue && regs <= kRegsCompute &&
         128 * c * kRegsCompute + 128 * kRegsIssue <= 128 * (c + 1) * regs;
}

// ---- shared-memory layout (bytes)
constexpr int kKeySlots = 4;
struct Smem {
  int b_off, key_off, ur_off, bar_off, total;
};
// What a CTA filters: lines of one axis, or of the two axes of its planes.
// finish() lays it out on the host: computed by each CTA it cost the launch
// about 0.1 us, which nothing hides (a CTA starts when the one before it has
// left the SM's shared memory).
struct Shape {
  int nd, pp, rep, axes;
  int half[2], kg[2];    // H, and 16-point blocks of it
  int stage;             // staging memory, bytes (aliases the A operands)
  int units, units_off;  // bytes for points' units behind it
  Smem lay;
  int cols, threads;     // TMEM columns
  int a_digit[2], b_half[2];   // bytes of a digit's A operand, of a half's table

  __host__ void finish() {
    int big = stage, bsum = 0, need = 0, blocks = 0;
    const bool res = nd == 4 || pp <= 8;   // tables of both halves resident, or one
    for (int i = 0; i < axes; ++i) {
      a_digit[i] = kLines * kg[i] * 32;
      b_half[i] = b_half_bytes(nd, kg[i]);
      const int a = nd * a_digit[i] * (both_halves(nd, kg[i]) ? 2 : 1);
      const int c = groups(nd) * group_cols(nd, kg[i]) * (dense_b(kg[i]) ? 2 : 1);
      big = a > big ? a : big;
      bsum += (res ? 2 : 1) * b_half[i];
      need = c > need ? c : need;
      blocks = kg[i] > blocks ? kg[i] : blocks;
    }
    for (int i = axes; i < 2; ++i) {
      a_digit[i] = a_digit[0];
      b_half[i] = b_half[0];
    }
    units_off = (big + 15) / 16 * 16;
    lay.b_off = (units_off + units + 127) / 128 * 128;
    lay.key_off = lay.b_off + bsum;
    lay.ur_off = lay.key_off + kKeySlots * kLines * 4;   // line keys
    lay.bar_off = lay.ur_off + 2 * kLines * 4;           // lines' units (planes: of both axes)
    lay.total = lay.bar_off + 64;                        // six mbarriers, TMEM address
    for (cols = 32; cols < need;) cols *= 2;
    threads = kLines * ((16 * blocks + pp * rep - 1) / (pp * rep)) + issuer_threads(pp);
  }
};

#ifdef __CUDACC__
// ---- tcgen05 / mbarrier wrappers
__device__ __forceinline__ uint32_t sm32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void tm_alloc(uint32_t slot, int cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tm_free(uint32_t base, int cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                        int accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.s32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Waits for phase `parity`, at most ~1 s of SM clocks; false on timeout.
__device__ __forceinline__ bool bar_wait(uint32_t bar, unsigned parity) {
  const long long t0 = clock64();
  while (true) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > 2000000000LL) return false;
  }
}
__device__ __forceinline__ void expect_bytes(uint32_t bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
// 1-D bulk copy global -> shared, counted on `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, unsigned bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
// Eight or four consecutive accumulator columns of this thread's lane.
__device__ __forceinline__ void tm_ld(uint32_t addr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(addr)
               : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tm_ld(uint32_t addr, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tm_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Unswizzled K-major operand: 8-row x 16-byte core matrices, `lbo` bytes
// between neighbours along K and `sbo` along M/N.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(lbo >> 4) << 16) |
         ((uint64_t)(sbo >> 4) << 32) | (1ULL << 46);
}

// ---- digits -> A operand.  Bytes of two neighbouring k become a half2 of
// 1024 + byte (exponent byte 0x64), minus 1152.
__device__ __forceinline__ uint32_t sub1152(uint32_t h2) {
  const __half2 v = *reinterpret_cast<const __half2 *>(&h2);
  const __half2 r = __hsub2(v, __half2half2(__ushort_as_half(0x6480)));
  return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ void bytes_to_f16(uint32_t wa, uint32_t wb, uint32_t (&d)[4]) {
  const uint32_t p = __byte_perm(wa, wb, 0x5140), q = __byte_perm(wa, wb, 0x7362);
  d[0] = sub1152(__byte_perm(p, 0x64646464u, 0x4140));   // byte 0 of a, b
  d[1] = sub1152(__byte_perm(p, 0x64646464u, 0x4342));
  d[2] = sub1152(__byte_perm(q, 0x64646464u, 0x4140));
  d[3] = sub1152(__byte_perm(q, 0x64646464u, 0x4342));
}
// digit pair words of two neighbouring k: out[digit], digit 0 the top one
__device__ __forceinline__ void digit_words(int64_t a, int64_t b, uint32_t (&o)[7]) {
  const uint64_t za = biased_digits(a), zb = biased_digits(b);
  uint32_t lo[4];
  bytes_to_f16((uint32_t)za, (uint32_t)zb, lo);
  const uint32_t ha = (uint32_t)(za >> 32), hb = (uint32_t)(zb >> 32);
  const uint32_t p = __byte_perm(ha, hb, 0x5140);
  o[0] = sub1152(__byte_perm(ha, hb, 0x7632) | 0x64006400u);
  o[1] = sub1152(__byte_perm(p, 0x64646464u, 0x4342));
  o[2] = sub1152(__byte_perm(p, 0x64646464u, 0x4140));
  o[3] = lo[3];
  o[4] = lo[2];
  o[5] = lo[1];
  o[6] = lo[0];
}
__device__ __forceinline__ void digit_words(int a, int b, uint32_t (&o)[4]) {
  uint32_t d[4];
  bytes_to_f16(biased_digits(a), biased_digits(b), d);
  o[0] = d[3];
  o[1] = d[2];
  o[2] = d[1];
  o[3] = d[0];
}

// ---- accumulators -> result
// 7 digits: sum_g D_g 256^(6-g) / 256 * 2^kFine, rounded.  D_g + 1.5*2^23 has the
// integer D_g in its low bits (|D_g| < 2^22).
__device__ __forceinline__ int64_t combine(const float (&D)[8]) {
  constexpr uint32_t C = 0x4B400000u;
  uint32_t I[8];
#pragma unroll
  for (int g = 0; g < 8; ++g) I[g] = __float_as_uint(D[g] + 12582912.f);
  const uint32_t p01 = I[0] * 256u + I[1] - C * 257u;
  const int p23 = (int)(I[2] * 256u + I[3] - C * 257u);
  const int p45 = (int)(I[4] * 256u + I[5] - C * 257u);
  const int p67 = (int)(I[6] * 256u + I[7] - C * 257u + (0x8000u >> kFine)) >> (16 - kFine);
  return (int64_t)((uint64_t)(p01 << kFine) << 32) + p67 + (int64_t)p45 * (1 << kFine) +
         (int64_t)p23 * (65536 << kFine);
}
__device__ __forceinline__ float combine(const float (&D)[4]) {
  return fmaf(fmaf(fmaf(D[0], 256.f, D[1]), 256.f, D[2]), 256.f, D[3]);
}

// mbarriers of a CTA
enum { kFull0 = 0, kFull1 = 1, kEmpty = 2, kDone0 = 3, kDone1 = 4, kTable = 5 };

// One CTA's filter engine.  ND digits, PP points per thread and half.  The
// last warp only issues the products: with one of the computing threads issuing
// them, its warp fell behind the others by the issue time of every round (36 %
// of all stalls at barriers at N = 128).  Computing warps signal digits written
// (full) and accumulators read (empty) once per warp and wait for products
// (done); none of it is a CTA-wide barrier.
template <int ND, int PP> struct Tile {
  typedef typename std::conditional<ND == 7, int64_t, int>::type I;
  typedef typename std::conditional<ND == 7, int64_t, float>::type Acc;

  unsigned char *smem;
  Smem lay;
  // per axis: blocks, H, bytes of a digit's A operand and of a half's table (no
  // arrays: an index at run time is a memory access)
  int kg0, kg1, half0, half1, ad0, ad1, bh0, bh1;
  const unsigned char *table;      // global (one axis): the digits of Kc, then of Kd
  int kg, H, a_digit, a_half, b_half, b_at;   // of the axis in hand
  int line, blk, rep, ln, warp, ncomp, cols;
  uint32_t tmem;
  unsigned phases;                 // parities of the products' barriers
  bool ok, both, issuer;
  static constexpr bool kSplit = ND == 7 && PP == 16;   // split_rows
  static constexpr bool kRes = ND == 4 || PP <= 8;   // both halves' tables resident
  static constexpr int NG = groups(ND);

  __device__ __forceinline__ uint32_t bar(int i) const { return sm32(smem + lay.bar_off) + 8 * i; }

  __device__ __forceinline__ void set_axis(int ax) {
    kg = ax ? kg1 : kg0;
    H = ax ? half1 : half0;
    both = both_halves(ND, kg);
    a_digit = ax ? ad1 : ad0;
    a_half = ND * a_digit;
    b_half = ax ? bh1 : bh0;
    b_at = ax ? 2 * bh0 : 0;
  }

  // Before the dependency wait: barriers, keys and the (constant) tables.
  __device__ __forceinline__ void setup(unsigned char *sm, const Shape &sh, const void *tab0,
                                        const void *tab1) {
    smem = sm;
    lay = sh.lay;
    cols = sh.cols;
    table = static_cast<const unsigned char *>(tab0) + sizeof(TcHead);
    kg0 = sh.kg[0];
    kg1 = sh.kg[1];
    half0 = sh.half[0];
    half1 = sh.half[1];
    ad0 = sh.a_digit[0];
    ad1 = sh.a_digit[1];
    bh0 = sh.b_half[0];
    bh1 = sh.b_half[1];
    set_axis(0);
    ncomp = blockDim.x - issuer_threads(PP);
    rep = PP == 4 ? sh.rep : 1;
    ln = kLines / rep;
    line = (threadIdx.x & 127) % ln;
    blk = (threadIdx.x & 127) / ln + rep * (threadIdx.x >> 7);
    warp = threadIdx.x >> 5;
    issuer = (int)threadIdx.x >= ncomp;
    phases = 0;
    ok = true;
    int *keys = reinterpret_cast<int *>(smem + lay.key_off);
    for (int i = threadIdx.x; i < kKeySlots * kLines; i += blockDim.x) keys[i] = 0;
    if ((int)threadIdx.x == ncomp) {
#pragma unroll
      for (int i = 0; i < 6; ++i)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar(i)),
                     "r"(i <= kEmpty ? ncomp / 32 : 1)
                     : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      if (kRes) {
        const unsigned b0 = 2 * bh0, b1 = sh.axes == 2 ? 2 * bh1 : 0;
        expect_bytes(bar(kTable), b0 + b1);
        bulk_load(sm32(smem + lay.b_off), table, b0, bar(kTable));
        if (b1)
          bulk_load(sm32(smem + lay.b_off) + b0,
                    static_cast<const unsigned char *>(tab1) + sizeof(TcHead), b1, bar(kTable));
      } else {
        load_half(0);
      }
    }
  }
  // The table of one half into the (free) B memory.
  __device__ __forceinline__ void load_half(int half) {
    expect_bytes(bar(kTable), bh0);
    bulk_load(sm32(smem + lay.b_off), table + half * bh0, bh0, bar(kTable));
  }
  // The issuing warp's part: after the dependency wait (a CTA that holds TMEM
  // must not wait for another one) TMEM, then `filters` filters, the f-th along
  // axis_of(f).
  template <typename F> __device__ __forceinline__ void run_issuer(int filters, F &&axis_of) {
    if (kSplit) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == ncomp / 32) tm_alloc(bar(6), cols);
    __syncthreads();
    read_tmem();
    if ((int)threadIdx.x == ncomp) {
      unsigned tphase = 0;
      for (int f = 0; f < filters; ++f) {
        set_axis(axis_of(f));
        for (int half = 0; half < 2; ++half) {
          wait_for(kFull0 + half, f & 1);
          if (!kRes || (f | half) == 0) wait_for(kTable, tphase++ & 1);
          fence_after();
          if (kSplit) {
            issue(half, 0);
            if (half == 1) {
              wait_for(kEmpty, f & 1);   // c's second round is read
              fence_after();
            }
            issue(half, 1);
          } else {
            issue(half, half);
          }
          if (!kRes && (half == 0 || f + 1 < filters)) {
            // the next half's table, once this half's products are done
            wait_for(kSplit ? kDone1 : kDone0 + half,
                     kSplit ? half : f & 1);
            if (ok) load_half(half ^ 1);
          }
        }
      }
    }
    __syncwarp();
  }
  // The computing threads' other side of it.
  __device__ __forceinline__ void run_compute() {
    if (kSplit) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsCompute));
  }
  // Every computing thread, once its loads are issued.
  __device__ __forceinline__ void start() {
    __syncthreads();
    read_tmem();
  }
  __device__ __forceinline__ void read_tmem() {
    fence_after();
    tmem = *reinterpret_cast<volatile uint32_t *>(smem + lay.bar_off + 48);
  }
  __device__ __forceinline__ void finish(unsigned *err) {
    if (!ok && err) atomicOr(err, 2u);
    __syncthreads();
    if (warp == ncomp / 32) tm_free(tmem, cols);
  }
  // barrier of the computing warps
  __device__ __forceinline__ void sync() const {
    asm volatile("bar.sync 1, %0;" ::"r"(ncomp) : "memory");
  }
  __device__ __forceinline__ void wait_for(int b, unsigned parity) {
    if (ok && !bar_wait(bar(b), parity)) ok = false;
  }
  __device__ __forceinline__ void signal(int b) {
    fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar(b)) : "memory");
  }
  // Accumulator buffer `buf` holds its products.
  __device__ __forceinline__ void wait_done(int buf) {
    wait_for(kDone0 + buf, phases >> buf & 1);
    phases ^= 1u << buf;
    fence_after();
    __syncwarp();
  }

  // digits of this thread's PP values (k = PP*blk + i) into A operand `half`
  __device__ __forceinline__ void put_digits(const I (&v)[PP], int half) {
    unsigned char *base = smem + (both ? half * a_half : 0) + line * 16;
    if (PP * blk < 16 * kg) {   // (planes: this axis may be shorter than the other one)
      constexpr int G = PP < 8 ? PP : 8;
#pragma unroll
      for (int h = 0; h < PP / G; ++h) {
        uint32_t w[G / 2][ND];
#pragma unroll
        for (int i = 0; i < G / 2; ++i) digit_words(v[G * h + 2 * i], v[G * h + 2 * i + 1], w[i]);
        const int k = PP * blk + G * h, bk = k / 8;
        unsigned char *dst =
            base + (dense_b(kg) ? bk : 2 * kg - 1 - bk) * (kLines * 16) + k % 8 * 2;
        for (int c = 0; c < (PP == 4 ? rep : 1); ++c) {
#pragma unroll
          for (int d = 0; d < ND; ++d) {
            if constexpr (G == 8)
              *reinterpret_cast<uint4 *>(dst + d * a_digit) =
                  make_uint4(w[0][d], w[1][d], w[2][d], w[3][d]);
            else
              *reinterpret_cast<uint2 *>(dst + d * a_digit) = make_uint2(w[0][d], w[1][d]);
          }
          dst += ln * 16;
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    signal(kFull0 + half);
  }

  // The digit products of half `half` (0: c, 1: d) into accumulator buffer
  // `buf` (also the round, where rows are split).  The block count is a constant
  // in each copy: with it read at run time an instruction took about 170 cycles
  // to issue among the computing warps, and 116 to run.
  __device__ __forceinline__ void issue(int half, int buf) {
    if (!ok) return;
    const uint32_t a0 = sm32(smem) + (both ? half * a_half : 0);
    const uint32_t b0 = sm32(smem + lay.b_off) + b_at + (kRes ? half * b_half : 0);
    switch (kg) {
      case 1: issue_kg<1>(a0, b0, buf); break;
      case 2: issue_kg<2>(a0, b0, buf); break;
      case 3: issue_kg<3>(a0, b0, buf); break;
      case 4: issue_kg<4>(a0, b0, buf); break;
      default: issue_shared(a0, b0); break;
    }
    mma_commit(bar(kDone0 + buf));
  }
  template <int KG> __device__ __forceinline__ void issue_kg(uint32_t a, uint32_t b, int buf) {
    if constexpr ((KG <= 2) == (PP <= 8)) {
      constexpr uint32_t gc = group_cols(ND, KG), id0 = (1u << 4) | ((kLines >> 4) << 24);
      constexpr uint32_t blbo = ND * gc * 16 * (kSplit ? 2 : 1), adig = kLines * KG * 32;
      const uint64_t ad = smem_desc(a, kLines * 16, 128);
      const uint64_t bd = smem_desc(b + (kSplit ? buf * ND * gc * 16 : 0), blbo, 128);
      const uint32_t d = tmem + buf * NG * gc;
#pragma unroll
      for (int s = 0; s < KG; ++s) {
        constexpr uint32_t kstep = 2 * kLines * 16 >> 4, bstep = 2 * blbo >> 4;
        const uint64_t as = ad + s * kstep, bs = bd + s * bstep;
        // K's first `rows` rows from row r0 on times x's digit i, from accumulator i on
        auto mma = [&](int i, uint32_t r0, uint32_t rows, int accumulate) {
          mma_f16(d + i * gc + r0, as + (i * adig >> 4), bs + r0, id0 | ((rows >> 3) << 17), accumulate);
        };
        // the first to write an accumulator overwrites it: with an eighth one, which
        // digit 0 does not meet, that is digit 1 for all but the first
        if (NG > ND && s == 0) {
          mma(1, 0, ND * gc, 0);
          mma(0, 0, gc, 0);
          mma(0, gc, (ND - 1) * gc, 1);
        }
#pragma unroll
        for (int i = NG > ND && s == 0 ? 2 : 0; i < ND; ++i)
          mma(i, 0, (NG - i < ND ? NG - i : ND) * gc, s + i != 0);
      }
    }
  }
  // lines above 128 points: one instruction per digit pair (see the top)
  __device__ __forceinline__ void issue_shared(uint32_t a, uint32_t b) {
    const uint32_t kp = 16 * kg, bdig = (4 * kg - 1) * 128;
    const uint32_t id = (1u << 4) | ((kLines >> 4) << 24) | ((kp >> 3) << 17);
    const uint64_t a0 = smem_desc(a, kLines * 16, 128), b0 = smem_desc(b, 128, 128);
#pragma unroll 1
    for (int s = 0; s < kg; ++s) {
      const uint64_t as = a0 + s * (2 * kLines * 16 >> 4), bs = b0 + s * (256 >> 4);
#pragma unroll
      for (int i = 0; i < ND; ++i)
#pragma unroll
        for (int j = 0; j < ND - i; ++j)
          mma_f16(tmem + (i + j) * kp, as + (uint32_t)(i * a_digit >> 4),
                  bs + (uint32_t)(j * bdig >> 4), id, (s | i) != 0);
    }
  }

  // GO outputs of this thread from accumulator buffer `buf`, starting at column
  // `col` of each group (with 16 points per thread four at a time: 32
  // accumulators in registers instead of 64, which spilled)
  static constexpr int GO = PP < 8 ? PP : 8;
  __device__ __forceinline__ void get(int buf, int col, Acc (&y)[GO]) {
    constexpr int L = PP == 16 ? 4 : GO;
    const uint32_t gc = group_cols(ND, kg);
    const uint32_t lane0 = tmem + ((uint32_t)(warp & 3) << 21);
    uint32_t addr = lane0 + (dense_b(kg) ? buf * NG * gc : 0) + col;
    if (col >= (int)gc) addr = lane0;   // (no such outputs: not used)
#pragma unroll
    for (int h = 0; h < GO; h += L) {
      float D[NG][L];
      __syncwarp();
#pragma unroll
      for (int g = 0; g < NG; ++g) tm_ld(addr + g * gc + h, D[g]);
      tm_wait_ld();
#pragma unroll
      for (int i = 0; i < L; ++i) {
        float d[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) d[g] = D[g][i];
        y[h + i] = combine(d);
      }
    }
  }

  // a = x[k], b = x[k+H] -> a = 2 y[k], b = 2 y[k+H] in the accumulators' units
  // (7 digits).
  // waiting() runs while the products do.
  template <typename G> __device__ __forceinline__ void filter(I (&a)[PP], I (&b)[PP], G &&waiting) {
    filter(a, b, waiting, [&](int i, I p, I q) {
      a[i] = p;
      b[i] = q;
    });
  }
  // ... -> out(i, 2 y[k], 2 y[k+H]).
  template <typename G, typename F>
  __device__ __forceinline__ void filter(I (&a)[PP], I (&b)[PP], G &&waiting, F &&out) {
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      const I s = a[i] + b[i];
      b[i] = a[i] - b[i];
      a[i] = s;
    }
    Acc c[PP], y[GO];
    put_digits(a, 0);
    if constexpr (ND == 7 && PP == 16) {
      // rounds c0 c1 d0 d1 (points 0-7, 8-15) in buffers 0 1 0 1: while one
      // buffer is read the other one's products run
      wait_done(0);
      get(0, 8 * blk, y);
#pragma unroll
      for (int i = 0; i < 8; ++i) c[i] = y[i];
      wait_done(1);          // c's products have read A
      put_digits(b, 1);
      get(1, 8 * blk, y);
#pragma unroll
      for (int i = 0; i < 8; ++i) c[8 + i] = y[i];
      signal(kEmpty);
      wait_done(0);
      get(0, 8 * blk, y);
#pragma unroll
      for (int i = 0; i < 8; ++i) out(i, c[i] + y[i], c[i] - y[i]);
      wait_done(1);
      get(1, 8 * blk, y);
#pragma unroll
      for (int i = 0; i < 8; ++i) out(8 + i, c[8 + i] + y[i], c[8 + i] - y[i]);
    } else {
      if (both) put_digits(b, 1);
      waiting();
      wait_done(0);
#pragma unroll
      for (int h = 0; h < PP / GO; ++h) {
        get(0, PP * blk + GO * h, y);
#pragma unroll
        for (int i = 0; i < GO; ++i) c[GO * h + i] = y[i];
      }
      if (!both) put_digits(b, 1);
      wait_done(1);
#pragma unroll
      for (int h = 0; h < PP / GO; ++h) {
        get(1, PP * blk + GO * h, y);
#pragma unroll
        for (int i = 0; i < GO; ++i) out(GO * h + i, c[GO * h + i] + y[i], c[GO * h + i] - y[i]);
      }
    }
    fence_before();
    __syncwarp();
  }

  // The largest of the line's keys over its threads; a barrier of the computing
  // warps.
  __device__ __forceinline__ int line_key(int slot, int key) {
    int *k = reinterpret_cast<int *>(smem + lay.key_off) + slot * kLines + line;
    atomicMax(k, key);
    sync();
    return *k;
  }
  // A slot for reuse two filters on (every thread has read it; by blk == 0).
  __device__ __forceinline__ void clear_key(int slot) {
    reinterpret_cast<int *>(smem + lay.key_off)[slot * kLines + line] = 0;
  }
  // Whether any computing thread says so; a barrier of the computing warps.
  __device__ __forceinline__ bool any(bool v) {
    int r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.s32 p, %2, 0;\n barrier.cta.red.or.pred q, 1, %1, p;\n"
        " selp.s32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"(ncomp), "r"(v ? 1 : 0)
        : "memory");
    return r != 0;
  }
};
#endif  // __CUDACC__

}  // namespace tc
}  // namespace scft
