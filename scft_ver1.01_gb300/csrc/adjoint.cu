// Derivatives of getConc (cuda_scft.cu:61-138): the box stress from the
// stored propagators, and the reverse-mode adjoint of the whole propagator
// march with contour checkpointing.  The reference has neither.
//
// Notation.  The two propagator chains of getConc form one chain of
// N = NsA + dNsB steps: q(0) = 1, q(s) = A_s q(s-1) (qA then qB), and the
// complementary chain q+(N) = 1, q+(s-1) = A_s q+(s) (q+B then q+A), with the
// split step A_s = W K W, W = exp(-w ds/2) of the block's field and K the
// diffusion filter exp(-ds k^2).  K is real, even and circulant, so A_s is
// symmetric and its adjoint is A_s itself.  Q = <q(N)>,
// phiA/B = (ds/Q) * contour sums (trapezoid or Simpson weights) of q q+ over
// the block's contour points.
//
// Box derivative of one step: dA_s/dL_a = W (dK/dL_a) W, where dK/dL_a is K
// with the axis-a gain multiplied by 2 ds k_a^2 / L_a (k_a ~ 1/L_a), or, for
// a length-1 axis (whose k is the constant 2 pi / L), the whole K times that
// factor.  Hence dQ/dL_a = (1/M) sum_s <q+(s), W (dK/dL_a) W q(s-1)>.
//
// dK/dL_a = K D_a with D_a along axis a alone, and K W q(s-1) = q(s) / W, so that
//   <q+(s), W (dK/dL_a) W q(s-1)> = <W^-1 D_a W q+(s), q(s)> :
// one pass an axis and step instead of one an axis for every axis.  The whole
// operator W K D_a W is applied where W or 1/W leaves 2^-60 .. 2^60, since the
// quotient could lose what q(s) has left, where W is rough (k_rough), since D_a
// without K multiplies the roundings of high wave numbers, and on axes that the
// tensor cores filter, which have the one table of K_a D_a.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "common.cuh"
#include "convert.cuh"
#include "ctx.h"

#define CK(call)                                                                        \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess)                                                              \
      return scft_fail(ctx, SCFT_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

#define CKL(call)                                                                       \
  do {                                                                                  \
    ++ctx->launches;                                                                    \
    CK(call);                                                                           \
  } while (0)

#define RC(call)                                                                        \
  do {                                                                                  \
    int rc_ = (call);                                                                   \
    if (rc_) return rc_;                                                                \
  } while (0)

namespace {

using scft::narrow;
using scft::widen;
constexpr int kT = 256;

int grid_for(long long n) {
  long long g = (n + kT - 1) / kT;
  return (int)std::min<long long>(g, 1 << 20);
}

// Two neighbouring points (grids have an even first axis).
template <typename R> struct alignas(2 * sizeof(R)) Two {
  R v[2];
};
template <typename R> __device__ __forceinline__ Two<R> two(const R *p) {
  return *reinterpret_cast<const Two<R> *>(p);
}
template <typename R> __device__ __forceinline__ void put(R *p, const Two<R> &x) {
  *reinterpret_cast<Two<R> *>(p) = x;
}
// acc1[b*nblk + blk] += sum_r a[b,r] * c1[b,r]  (and acc2 with c2).  Every (b, blk)
// slot has one writer, so repeated calls accumulate in a fixed order
// (bit-reproducible).
template <typename R, typename S>
__global__ void k_dot_acc(const R *__restrict__ a, long long a_bs, const S *__restrict__ c1,
                          long long c1_bs, const S *__restrict__ c2, long long c2_bs,
                          long long M, double *__restrict__ acc1, double *__restrict__ acc2) {
  __shared__ double sh[kT / 2];
  const long long b = blockIdx.y;
  const int nblk = gridDim.x;
  double v1 = 0.0, v2 = 0.0;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < M;
       r += (long long)nblk * blockDim.x) {
    const double x = widen(a[b * a_bs + r]);
    v1 += x * widen(c1[b * c1_bs + r]);
    if (c2) v2 += x * widen(c2[b * c2_bs + r]);
  }
  v1 = scft::block_sum<kT>(v1, sh);
  if (threadIdx.x == 0) acc1[b * nblk + blockIdx.x] += v1;
  if (c2) {
    v2 = scft::block_sum<kT>(v2, sh);
    if (threadIdx.x == 0) acc2[b * nblk + blockIdx.x] += v2;
  }
}

// acc[k][blk] += sum_{r < n} x[k][r] * y[r] for N arrays x.  The FP64 pipe bounds it
// (two operations a product of double-float values, y converted once for all), or
// HBM: two points a load and U loads of each array in flight.  Its blocks do not
// follow the grid's size: 64 slices of 30 x 16 x 32 on the 15 blocks of a single
// slice took 52 us.
constexpr int kDotBlocks = 3 * 152;
template <typename R> struct DotArgs {
  const R *x[4];
  double *acc[4];
  int n;
};
template <typename R, int N, int U>
__global__ void __launch_bounds__(kT) k_dots(DotArgs<R> d, const R *__restrict__ y, long long n) {
  __shared__ double sh[kT / 2];
  double v[N][2] = {};
  const long long S = 2 * (long long)gridDim.x * blockDim.x;
  for (long long r0 = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x); r0 < n; r0 += U * S) {
    Two<R> tx[U][N], ty[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r0 + u * S < n) {
        ty[u] = two(y + (r0 + u * S));
#pragma unroll
        for (int k = 0; k < N; ++k) tx[u][k] = two(d.x[k] + (r0 + u * S));
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r0 + u * S < n) {
        const double y0 = widen(ty[u].v[0]), y1 = widen(ty[u].v[1]);
#pragma unroll
        for (int k = 0; k < N; ++k) {
          v[k][0] = fma(widen(tx[u][k].v[0]), y0, v[k][0]);
          v[k][1] = fma(widen(tx[u][k].v[1]), y1, v[k][1]);
        }
      }
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double s = scft::block_sum<kT>(v[k][0] + v[k][1], sh);
    if (threadIdx.x == 0) d.acc[k][blockIdx.x] += s;
  }
}

// out = 1 / W
__device__ __forceinline__ float inverse(float w) { return 1.0f / w; }
__device__ __forceinline__ double inverse(double w) { return 1.0 / w; }
__device__ __forceinline__ scft::dfloat inverse(scft::dfloat w) {
  return scft::dfloat(1.0 / (double)w);
}
template <typename R>
__global__ void k_inverse(const R *__restrict__ W, R *__restrict__ out, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = inverse(W[i]);
}
// *flag is set where W is not within 2^-60 .. 2^60, or where D_a W^2, by second
// differences (c[a] = 2 ds / L_a (n_a / L_a)^2; 0: not asked), is above kRough of W^2
// itself.  Fields of a solve come to 0.001 - 0.02 (smooth patterns, or noise of 0.02 on
// them); with noise of +-15 they come to 5, and the quotient's stress was 25 - 250 times
// further off than the whole operator's (64^3: FP32 1.1e-5 against 3.9e-7, double-float
// 4.9e-13 against 1.9e-15), in proportion to it.
constexpr float kRough = 0.05f;
__device__ __forceinline__ float approx(float w) { return w; }
__device__ __forceinline__ float approx(double w) { return (float)w; }
__device__ __forceinline__ float approx(scft::dfloat w) { return w.hi; }
struct Axes {
  int n[3];
  float c[3];
};
template <typename R>
__global__ void k_rough(const R *__restrict__ W, Axes g, long long n, int *__restrict__ flag) {
  bool bad = false;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float w = approx(W[i]);
    bad |= !(w > 0x1p-60f && w < 0x1p60f);
    long long at = i, st = 1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int m = g.n[a], k = (int)(at % m);
      if (g.c[a] != 0.0f) {
        const float up = approx(W[k + 1 < m ? i + st : i - (m - 1) * st]);
        const float dn = approx(W[k > 0 ? i - st : i + (m - 1) * st]);
        bad |= !(g.c[a] * fabsf(up * up + dn * dn - 2.0f * w * w) <= kRough * w * w);
      }
      at /= m;
      st *= m;
    }
  }
  if (bad) *flag = 1;
}

// out[b] = sum_k partial[b*nblk + k]
__global__ void k_sum_slots(const double *__restrict__ partial, int nblk, double *__restrict__ out) {
  __shared__ double sh[kT / 2];
  const int b = blockIdx.x;
  double v = 0.0;
  for (int k = threadIdx.x; k < nblk; k += blockDim.x) v += partial[(long long)b * nblk + k];
  v = scft::block_sum<kT>(v, sh);
  if (threadIdx.x == 0) out[b] = v;
}

// One contour point's weights in the accumulators of sums of q q+ (S: the density
// sums; G: the sums of the Q part, Simpson only) and in the adjoint seed.  How they
// are used is decided on the host: comparisons of doubles take the FP64 pipe too.
enum { kNone = 0, kOne = 1, kSome = 2 };   // weight 0 (arrays not touched), 1, other
struct Point {
  double c[2], g[2];          // blocks A, B
  int cm[2], gm[2], in;       // in: the block that the point lies inside of, or -1
  double *S[2], *G[2];
  const double *pb[2];        // ffl * phibar
};
// the point's seed, (cA phibarA + cB phibarB) ffl
__device__ __forceinline__ void seed_at(const Point &pt, long long o, double (&s)[2]) {
  s[0] = s[1] = 0.0;
#pragma unroll
  for (int f = 0; f < 2; ++f)
    if (pt.cm[f]) {
      const Two<double> b = two(pt.pb[f] + o);
      if (pt.cm[f] == kOne) {   // (within a block, where the other one's weight is 0)
        s[0] = b.v[0];
        s[1] = b.v[1];
      } else {
        s[0] += pt.c[f] * b.v[0];
        s[1] += pt.c[f] * b.v[1];
      }
    }
}
// the accumulators of a point, read before anything is written; then with q q+ added
struct Sums {
  Two<double> s[2], g[2];
};
__device__ __forceinline__ void load_sums(const Point &pt, long long o, Sums &u) {
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    if (pt.cm[f]) u.s[f] = two(pt.S[f] + o);
    if (pt.gm[f]) u.g[f] = two(pt.G[f] + o);
  }
}
__device__ __forceinline__ void add_sum(double *acc, Two<double> &a, int mode, double c,
                                        const double (&x)[2], const double (&y)[2]) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (mode == kOne) a.v[k] = fma(x[k], y[k], a.v[k]);
    else a.v[k] += c * (x[k] * y[k]);
  }
  put(acc, a);
}
__device__ __forceinline__ void store_sums(const Point &pt, long long o, Sums &u,
                                           const double (&x)[2], const double (&y)[2]) {
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    if (pt.cm[f]) add_sum(pt.S[f] + o, u.s[f], pt.cm[f], pt.c[f], x, y);
    if (pt.gm[f]) add_sum(pt.G[f] + o, u.g[f], pt.gm[f], pt.g[f], x, y);
  }
}

// out = c[b] * in
__global__ void k_scale(double *__restrict__ out, const double *__restrict__ in,
                        const double *__restrict__ c, long long M) {
  const long long b = blockIdx.y;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += (long long)gridDim.x * blockDim.x)
    out[b * M + i] = c[b] * in[b * M + i];
}

// The end point of a chain: the adjoint seed there; with q also its sums (q+ = 1).
template <typename R>
__global__ void k_seed(Point pt, R *__restrict__ out, const R *__restrict__ q, long long q_bs,
                       long long M) {
  const long long b = blockIdx.y;
  for (long long i = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x); i < M;
       i += 2 * (long long)gridDim.x * blockDim.x) {
    const long long o = b * M + i;
    double s[2];
    seed_at(pt, o, s);
    Two<R> r;
    r.v[0] = (R)s[0];
    r.v[1] = (R)s[1];
    put(out + o, r);
    if (q) {
      Sums u;
      load_sums(pt, o, u);
      const Two<R> x = two(q + b * q_bs + i);
      const double xx[2] = {widen(x.v[0]), widen(x.v[1])}, one[2] = {1.0, 1.0};
      store_sums(pt, o, u, xx, one);
    }
  }
}

// One step of a reverse sweep.  Over the q chain, s -> s-1 (SUMS; a = lam, x1 = q(s),
// x0 = q(s-1), y = q+(s-1)), with the sums at s-1; over the q+ chain, s-1 -> s
// (a = mu, x1 = q+(s-1), x0 = q+(s), y = q(s)):
//   wbar += a x1 + (A a) x0                        (field of step s; the caller's -ds/2)
//   a_out = A a + ffl (cA phibarA + cB phibarB) y    at the point reached
// FP64 pipe and memory latency bound it: with the sums of the Q part taken from the
// density sums (trapezoid: one is twice the other), only the block's own arrays
// touched, the constant factors outside and conversions in integers it has 4 FP64
// operations a point instead of 19 and moves 64 bytes instead of 108, all loads first
// (64^3: 8.4 us with 8 operations, 12.6 with 16).
// INNER: the point lies inside block pt.in, with weight 1 (trapezoid).
template <typename R, bool SUMS, bool INNER>
__global__ void __launch_bounds__(kT)
    k_sweep(Point pt, const R *__restrict__ p, const R *__restrict__ a, const R *__restrict__ x1_,
            long long x1_bs, const R *__restrict__ x0_, long long x0_bs, const R *__restrict__ y_,
            double *__restrict__ wbar, R *__restrict__ a_out, long long M) {
  scft::pdl_wait();
  scft::pdl_release();
  const long long b = blockIdx.y;
  for (long long i = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x); i < M;
       i += 2 * (long long)gridDim.x * blockDim.x) {
    const long long o = b * M + i;
    const Two<R> tp = two(p + o), ta = two(a + o), t1 = two(x1_ + b * x1_bs + i),
                 t0 = two(x0_ + b * x0_bs + i), ty = two(y_ + o);
    Two<double> w = two(wbar + o);
    Sums u;
    double s[2], x0[2], y[2];
    if constexpr (INNER) {
      if (SUMS) u.s[0] = two(pt.S[pt.in] + o);
      const Two<double> sd = two(pt.pb[pt.in] + o);
      s[0] = sd.v[0];
      s[1] = sd.v[1];
    } else {
      if (SUMS) load_sums(pt, o, u);
      seed_at(pt, o, s);
    }
    Two<R> out;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double pp = widen(tp.v[k]);
      x0[k] = widen(t0.v[k]);
      y[k] = widen(ty.v[k]);
      w.v[k] = fma(pp, x0[k], fma(widen(ta.v[k]), widen(t1.v[k]), w.v[k]));
      narrow(fma(s[k], y[k], pp), out.v[k]);
    }
    put(wbar + o, w);
    put(a_out + o, out);
    if constexpr (SUMS && INNER) add_sum(pt.S[pt.in] + o, u.s[0], kOne, 1.0, x0, y);
    else if constexpr (SUMS) store_sums(pt, o, u, x0, y);
  }
}

// wbar = -hds wbar + coef[b] * G
__global__ void k_finish(double *__restrict__ wbar, const double *__restrict__ G, double hds,
                         const double *__restrict__ coef, long long M) {
  const long long b = blockIdx.y;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += (long long)gridDim.x * blockDim.x)
    wbar[b * M + i] = coef[b] * G[b * M + i] - hds * wbar[b * M + i];
}


}  // namespace

// Work buffers of the adjoint and the stress (working precision R unless
// noted), allocated on first use and kept for later calls.
struct AdjointState {
  size_t bytes = 0;
  void *mem = nullptr;          // one allocation, carved below
  int K = 0, nck1 = 0, nck2 = 0;
  std::vector<int> pos1, pos2;  // checkpoint positions: q at s = pos1[j], q+ at s = N - pos2[j]
  void *ck1 = nullptr, *ck2 = nullptr, *seg = nullptr;
  void *v[12] = {};             // [B][M] vectors
  double *d[10] = {};           // [B][M] FP64 accumulators and seeds
  double *acc = nullptr;        // [kinds][B][nblk]
  double *small = nullptr;      // [8][B]
  // stress chunk buffers
  size_t sbytes = 0, sacc_off = 0;
  void *smem = nullptr;          // chunk x 3 slices, 1/W, then reduction slots
  int chunk = 0;
};

void scft_internal_adjoint_free(scft_ctx *ctx) {
  if (!ctx->adj) return;
  cudaFree(ctx->adj->mem);
  cudaFree(ctx->adj->smem);
  delete ctx->adj;
  ctx->adj = nullptr;
}

namespace {

constexpr int kAccKinds = 16;
enum AccKind { ACC_L1 = 0, ACC_Q = 3, ACC_L2 = 6, ACC_U1 = 9, ACC_UQ = 10, ACC_U2 = 11,
               ACC_FFL = 12 };

int field_of_step(const scft_ctx *ctx, int s) { return s <= ctx->NsA ? 0 : 1; }

// contour weights of point s in the A and B blocks (those of the forward
// contour sums: trapezoid, or Simpson with SCFT_FLAG_SIMPSON)
void weights(const scft_ctx *ctx, int s, double *cA, double *cB) {
  const bool simpson = (ctx->p.flags & SCFT_FLAG_SIMPSON) != 0;
  *cA = s <= ctx->NsA ? scft::contour_weight(s, ctx->NsA, simpson) : 0.0;
  *cB = s >= ctx->NsA ? scft::contour_weight(s - ctx->NsA, ctx->dNsB, simpson) : 0.0;
}

int ensure_adjoint(scft_ctx *ctx, int K) {
  const int N = ctx->NsA + ctx->dNsB;
  const long long M = ctx->M, B = ctx->batch;
  const size_t rb = ctx->rbytes;
  if (!ctx->adj) ctx->adj = new AdjointState();
  AdjointState &A = *ctx->adj;
  if (A.mem && A.K == K) return SCFT_OK;
  cudaFree(A.mem);
  A.mem = nullptr;
  A.K = K;
  A.pos1.clear();
  for (int s = 0; s < N; s += K) A.pos1.push_back(s);
  A.pos1.push_back(N);
  A.pos2 = A.pos1;      // q+ checkpoints at distance t from the chain end
  A.nck1 = A.nck2 = (int)A.pos1.size();
  const size_t slice = (size_t)M * B * rb;
  const size_t dslice = (size_t)M * B * 8;
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  size_t need = up(slice * A.nck1) + up(slice * A.nck2) + up((size_t)(K + 1) * slice) +
                12 * up(slice) + 10 * up(dslice) + up(8 * (size_t)kAccKinds * B * ctx->nblk) +
                up(8 * (8 + (size_t)kAccKinds) * B);
  CK(cudaMalloc(&A.mem, need));
  A.bytes = need;
  unsigned char *m = static_cast<unsigned char *>(A.mem);
  size_t off = 0;
  auto take = [&](size_t n) { void *p = m + off; off += up(n); return p; };
  A.ck1 = take(slice * A.nck1);
  A.ck2 = take(slice * A.nck2);
  A.seg = take((size_t)(K + 1) * slice);
  for (int i = 0; i < 12; ++i) A.v[i] = take(slice);
  for (int i = 0; i < 10; ++i) A.d[i] = static_cast<double *>(take(dslice));
  A.acc = static_cast<double *>(take(8 * (size_t)kAccKinds * B * ctx->nblk));
  A.small = static_cast<double *>(take(8 * (8 + (size_t)kAccKinds) * B));
  return SCFT_OK;
}

// Whether axis pass pi takes W K D_a W.
bool whole_axis(const scft_ctx *ctx, int pi, int wide) { return wide || ctx->passes[pi].tc; }
// ... for all of them: the FFT axes too, where these factors do not allow the quotient
// (flag: device scratch).
template <typename R>
int whole_wanted(scft_ctx *ctx, const R *const (&W)[2], int *flag, int *wide) {
  const double L[3] = {ctx->p.lx, ctx->p.ly, ctx->p.lz};
  cudaStream_t st = ctx->st;
  Axes g = {{ctx->p.nx, ctx->p.ny, ctx->p.nz}, {0.0f, 0.0f, 0.0f}};
  *wide = 1;
  for (size_t pi = 0; pi < ctx->passes.size(); ++pi) {
    if (ctx->passes[pi].tc) continue;
    const int a = ctx->pass_axis[pi];
    g.c[a] = (float)(2.0 * ctx->p.ds0 / L[a] * (g.n[a] / L[a]) * (g.n[a] / L[a]));
    *wide = 0;
  }
  if (*wide) return SCFT_OK;
  CK(cudaMemsetAsync(flag, 0, sizeof(int), st));
  for (int f = 0; f < 2; ++f) {
    k_rough<R><<<grid_for(ctx->M * ctx->batch), kT, 0, st>>>(W[f], g, ctx->M * ctx->batch, flag);
    ++ctx->launches;
  }
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(wide, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return SCFT_OK;
}
// out = W K D_a W in, a the axis of pass pi (s0, s1: scratch).
template <typename R>
int whole_term(scft_ctx *ctx, int pi, const R *in, long long in_bs, const R *W, long long w_bs,
               int nb, R *out, R *s0, R *s1, cudaStream_t st) {
  return scft_internal_filter(ctx, in, in_bs, out, ctx->M, W, W, w_bs, nb, pi, s0, s1, st);
}

template <typename R>
int adjoint_impl(scft_ctx *ctx, const double *h_pbA, const double *h_pbB, const double *h_Qbar,
                 double *h_wabar, double *h_wbbar, double *h_Lbar) {
  AdjointState &A = *ctx->adj;
  const long long M = ctx->M;
  const int B = ctx->batch, N = ctx->NsA + ctx->dNsB, nblk = ctx->nblk, K = A.K;
  const double ds = ctx->p.ds0, hds = ds / 2;
  cudaStream_t st = ctx->st;
  const bool want_L = h_Lbar != nullptr;
  const int np = (int)ctx->passes.size();
  bool has_unit = false;
  for (int a = 0; a < 3; ++a) has_unit |= ctx->unit_c[a] != 0.0;

  R *ck1 = static_cast<R *>(A.ck1), *ck2 = static_cast<R *>(A.ck2);
  R *seg = static_cast<R *>(A.seg);
  R *W[2] = {static_cast<R *>(A.v[0]), static_cast<R *>(A.v[1])};
  R *va = static_cast<R *>(A.v[2]), *vb = static_cast<R *>(A.v[3]);    // marching pairs
  R *x = static_cast<R *>(A.v[4]), *y = static_cast<R *>(A.v[5]);
  R *l0 = static_cast<R *>(A.v[6]), *l1 = static_cast<R *>(A.v[7]);    // adjoint pair
  R *p = static_cast<R *>(A.v[8]), *t = static_cast<R *>(A.v[9]);
  R *s0 = static_cast<R *>(A.v[10]), *s1 = static_cast<R *>(A.v[11]);
  void *scratch[scft::kStepSet] = {s0, s1, t};
  double *wa_avg = A.d[0], *wbar[2] = {A.d[1], A.d[2]}, *G[2] = {A.d[3], A.d[4]};
  double *S[2] = {A.d[5], A.d[6]}, *pb[2] = {A.d[7], A.d[8]}, *pbs[2] = {A.d[0], A.d[9]};
  double *acc = A.acc;
  double *Q = A.small, *ffl = A.small + B, *sum = A.small + 2 * B, *coef = A.small + 3 * B;
  double *sums = A.small + 8 * B;   // [kinds][B]
  const long long ckbs1 = (long long)A.nck1 * M, ckbs2 = (long long)A.nck2 * M;
  const long long segbs = (long long)(K + 1) * M;
  const size_t dbytes = sizeof(double) * M * B;
  auto accp = [&](int kind) { return acc + (size_t)kind * B * nblk; };

  // ---- inputs: getConc's mean-free wA (cuda_scft.cu:71), Boltzmann factors, seeds
  CKL(scft::launch_copy_slice<double>(wa_avg, M, ctx->wa, M, M, B, st));
  CKL(scft::launch_partial_sum<double>(wa_avg, M, M, B, ctx->partial, nblk, st));
  CKL(scft::launch_finalize_sum(ctx->partial, nblk, B, 1.0, sum, st));
  CKL(scft::launch_minus_average(wa_avg, sum, M, B, st));
  CKL(scft::launch_boltzmann<R>(wa_avg, W[0], M * B, hds, st));
  CKL(scft::launch_boltzmann<R>(ctx->wb, W[1], M * B, hds, st));
  const double *h_pb[2] = {h_pbA, h_pbB};
  for (int f = 0; f < 2; ++f) {
    if (h_pb[f]) CK(cudaMemcpyAsync(pb[f], h_pb[f], dbytes, cudaMemcpyHostToDevice, st));
    else CK(cudaMemsetAsync(pb[f], 0, dbytes, st));
  }
  for (double *z : {wbar[0], wbar[1], G[0], G[1], S[0], S[1]}) CK(cudaMemsetAsync(z, 0, dbytes, st));
  CK(cudaMemsetAsync(acc, 0, sizeof(double) * kAccKinds * B * nblk, st));

  // Steps that do not depend on each other run as one set of launches: the two
  // chains' forward marches, and in a sweep the companion chain, the adjoint and
  // the next segment's recomputation: 3 N steps in sequence instead of 8 N, with
  // two launches each where the x and y passes share one.  What bounds it is the
  // launches in sequence (about 4 us each at 64^3).  N = 200 steps, ms a call:
  // FP32 32^3 12.0 -> 5.0, 64^3 16.9 -> 7.7, 128 x 128 x 64 41.5 -> 17.8; FP64 64^3
  // 118 -> 24.
  StepIO io[scft::kStepSet];
  int nio = 0;
  auto add = [&](const R *in, long long in_bs, R *out, long long out_bs, int f) {
    io[nio++] = StepIO{in, W[f], out, in_bs, out_bs};
  };
  auto run = [&]() {
    const int n = nio;
    nio = 0;
    return scft_internal_steps(ctx, io, n, M, B, scratch, st);
  };
  const dim3 eg(grid_for(M), B), eg2(grid_for(M / 2), B);

  // ---- segments between checkpoints, in the order the sweeps take them.  Of a
  // segment's slices 0 .. len the first and the last are checkpoints; the others
  // lie in seg, upwards from its first slot or downwards from its last one, in
  // turn: the next segment grows into the slots the present one has left behind.
  struct Segm { const R *ck; long long ckbs; int chain, j, lo, len; };
  std::vector<Segm> segs;
  for (int c = 0; c < 2; ++c) {
    const std::vector<int> &pos = c == 0 ? A.pos1 : A.pos2;
    for (int j = (int)pos.size() - 2; j >= 0; --j)
      segs.push_back(Segm{c == 0 ? ck1 : ck2, c == 0 ? ckbs1 : ckbs2, c, j, pos[j],
                          pos[j + 1] - pos[j]});
  }
  auto slice = [&](size_t i, int k, long long *bs) -> R * {
    const Segm &g = segs[i];
    if (k == 0 || k == g.len) {
      *bs = g.ckbs;
      return const_cast<R *>(g.ck) + (long long)(g.j + (k ? 1 : 0)) * M;
    }
    *bs = segbs;
    return seg + (long long)(i & 1 ? K + 1 - k : k - 1) * M;
  };
  // the step of a chain from its distance u-1 to u: q(u-1) -> q(u), q+(s) -> q+(s-1)
  auto step_of = [&](int chain, int u) { return chain == 0 ? u : N - u + 1; };
  auto recompute = [&](size_t i, int k) {   // slice k of segment i
    long long ibs, obs;
    const R *in = slice(i, k - 1, &ibs);
    R *out = slice(i, k, &obs);
    add(in, ibs, out, obs, field_of_step(ctx, step_of(segs[i].chain, segs[i].lo + k)));
  };

  // ---- forward: checkpoints of both chains every K steps; the q chain's last
  // segment straight into its slots
  CKL(scft::launch_fill<R>(ck1, M, R(1), ckbs1, B, st));
  CKL(scft::launch_fill<R>(ck2, M, R(1), ckbs2, B, st));
  {
    const R *cur[2] = {ck1, ck2};
    long long cur_bs[2] = {ckbs1, ckbs2};
    R *ck[2] = {ck1, ck2}, *pair[2][2] = {{va, vb}, {x, y}};
    const long long ckbs[2] = {ckbs1, ckbs2};
    size_t j = 1;
    for (int u = 1; u <= N; ++u) {
      const bool at = j < A.pos1.size() && A.pos1[j] == u;   // (pos1 and pos2 are the same)
      for (int c = 0; c < 2; ++c) {
        long long bs = M;
        R *dst = cur[c] == pair[c][0] ? pair[c][1] : pair[c][0];
        if (at) {
          dst = ck[c] + (long long)j * M;
          bs = ckbs[c];
        } else if (c == 0 && u > segs[0].lo) {
          dst = slice(0, u - segs[0].lo, &bs);
        }
        add(cur[c], cur_bs[c], dst, bs, field_of_step(ctx, step_of(c, u)));
        cur[c] = dst;
        cur_bs[c] = bs;
      }
      RC(run());
      if (at) ++j;
    }
  }
  // Q = <q(N)>, ffl = ds/Q (cal_ql and getConc's host lines, cuda_scft.cu:118-125)
  const R *qN = ck1 + (long long)(A.nck1 - 1) * M;
  CKL(scft::launch_partial_sum<R>(qN, ckbs1, M, B, ctx->partial, nblk, st));
  CKL(scft::launch_finalize_sum(ctx->partial, nblk, B, 1.0, sum, st));
  CKL(scft::launch_q_ffl(sum, M, ds, B, Q, ffl, st));
  for (int f = 0; f < 2; ++f) {
    k_scale<<<eg, kT, 0, st>>>(pbs[f], pb[f], ffl, M);
    ++ctx->launches;
  }
  CK(cudaGetLastError());

  auto dot = [&](const R *a, long long a_bs, const R *c1, long long c1_bs, const R *c2,
                 long long c2_bs, double *acc1, double *acc2) {
    k_dot_acc<R, R><<<dim3(nblk, B), kT, 0, st>>>(a, a_bs, c1, c1_bs, c2, c2_bs, M, acc1, acc2);
    ++ctx->launches;
    return cudaGetLastError();
  };
  // The sum over a block's steps of q+(s) q(s) + q+(s-1) q(s-1) is twice its
  // trapezoid sum: S itself, or G beside Simpson's S.
  const bool simpson = (ctx->p.flags & SCFT_FLAG_SIMPSON) != 0;
  auto point = [&](int s, bool sums) {
    Point pt;
    weights(ctx, s, &pt.c[0], &pt.c[1]);
    const int n[2] = {ctx->NsA, ctx->dNsB};
    pt.in = -1;
    for (int f = 0; f < 2; ++f) {
      const int at = f == 0 ? s : s - ctx->NsA;
      pt.g[f] = sums && simpson ? scft::contour_weight(at, n[f], false) : 0.0;
      auto mode = [](double w) { return w == 0.0 ? kNone : (w == 1.0 ? kOne : kSome); };
      pt.cm[f] = mode(pt.c[f]);
      pt.gm[f] = mode(pt.g[f]);
      pt.S[f] = S[f];
      pt.G[f] = G[f];
      pt.pb[f] = pbs[f];
      if (!simpson && pt.cm[f] == kOne) pt.in = f;   // (the other block's weight is 0)
    }
    return pt;
  };

  // the box derivatives' 1/W (the marching pair is free), where it will do
  R *Winv[2] = {va, vb};
  int wide = 0;
  if (want_L) {
    const R *const Wc[2] = {W[0], W[1]};
    RC(whole_wanted<R>(ctx, Wc, reinterpret_cast<int *>(A.small + 4 * B), &wide));
    for (int f = 0; f < 2 && !wide; ++f) {
      k_inverse<R><<<grid_for(M * B), kT, 0, st>>>(W[f], Winv[f], M * B);
      ++ctx->launches;
    }
    CK(cudaGetLastError());
  }

  // ---- the sweeps: the q chain's in reverse (s = N .. 1, q+ marched alongside),
  // then the q+ chain's (s = 1 .. N, q marched alongside)
  R *a = l0, *a_n = l1, *co = x, *co_n = y;   // adjoint, companion chain
  for (size_t i = 0; i < segs.size(); ++i) {
    const Segm &g = segs[i];
    const bool q_chain = g.chain == 0, more = i + 1 < segs.size();
    if (i == 0 || segs[i - 1].chain != g.chain) {
      k_seed<R><<<eg2, kT, 0, st>>>(point(q_chain ? N : 0, q_chain), a, q_chain ? qN : nullptr,
                                    ckbs1, M);
      ++ctx->launches;
      CK(cudaGetLastError());
      CKL(scft::launch_fill<R>(co, M * B, R(1), 0, 1, st));
    }
    for (int k = g.len; k >= 1; --k) {
      const int s = step_of(g.chain, g.lo + k), f = field_of_step(ctx, s);
      long long bs1, bs0;
      const R *x1 = slice(i, k, &bs1), *x0 = slice(i, k - 1, &bs0);
      add(co, M, co_n, M, f);                  // q+(s-1) / q(s)
      add(a, M, p, M, f);                      // A a
      const int rec = g.len - k + 1;
      if (more && rec < segs[i + 1].len) recompute(i + 1, rec);
      RC(run());
      if (want_L) {
        const int L = q_chain ? ACC_L1 : ACC_L2;
        for (int pi = 0; pi < np; ++pi) {
          const bool whole = whole_axis(ctx, pi, wide);
          if (whole)   // <a, W K D W x0>
            RC(whole_term<R>(ctx, pi, x0, bs0, W[f], M, B, t, s0, s1, st));
          else         // = <A a, W^-1 D W x0>
            RC(scft_internal_deriv(ctx, pi, x0, bs0, t, M, W[f], Winv[f], M, B, st));
          CK(dot(t, M, whole ? a : p, M, q_chain ? (whole ? co : co_n) : nullptr, M, accp(L + pi),
                 q_chain ? accp(ACC_Q + pi) : nullptr));
        }
        if (has_unit)
          CK(dot(x1, bs1, a, M, q_chain ? co : nullptr, M, accp(q_chain ? ACC_U1 : ACC_U2),
                 q_chain ? accp(ACC_UQ) : nullptr));
      }
      const Point pt = point(q_chain ? s - 1 : s, q_chain);
      auto k_step = pt.in >= 0 ? (q_chain ? k_sweep<R, true, true> : k_sweep<R, false, true>)
                               : (q_chain ? k_sweep<R, true, false> : k_sweep<R, false, false>);
      CKL(scft::launch_pdl(k_step, eg2, dim3(kT), 0, st, pt,
                           p, a, x1, bs1, x0, bs0, co_n, wbar[f], a_n, M));
      std::swap(a, a_n);
      std::swap(co, co_n);
    }
    for (int rec = g.len + 1; more && rec < segs[i + 1].len; ++rec) {
      recompute(i + 1, rec);
      RC(run());
    }
  }
  // ---- the Q part: Qbar_tot = Qbar - fflbar ds / Q^2, fflbar = <phibar, S>
  k_dot_acc<double, double><<<dim3(nblk, B), kT, 0, st>>>(pb[0], M, S[0], M, nullptr, 0, M,
                                                          accp(ACC_FFL), nullptr);
  k_dot_acc<double, double><<<dim3(nblk, B), kT, 0, st>>>(pb[1], M, S[1], M, nullptr, 0, M,
                                                          accp(ACC_FFL), nullptr);
  ctx->launches += 2;
  CK(cudaGetLastError());
  std::vector<double> sums_h((size_t)kAccKinds * B), hQ(B);
  k_sum_slots<<<kAccKinds * B, kT, 0, st>>>(acc, nblk, sums);
  ++ctx->launches;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(sums_h.data(), sums, 8 * (size_t)kAccKinds * B, cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(hQ.data(), Q, 8 * B, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  std::vector<double> qtot(B), cf(2 * B);
  for (int b = 0; b < B; ++b) {
    const double fflbar = sums_h[(size_t)ACC_FFL * B + b];
    qtot[b] = (h_Qbar ? h_Qbar[b] : 0.0) - fflbar * ds / (hQ[b] * hQ[b]);
    cf[b] = -ds * qtot[b] / (double)M;   // (2 S: see point)
  }
  CK(cudaMemcpyAsync(coef, cf.data(), 8 * B, cudaMemcpyHostToDevice, st));
  for (int f = 0; f < 2; ++f) {
    if ((f == 0 ? ctx->NsA : ctx->dNsB) == 0) continue;
    k_finish<<<eg, kT, 0, st>>>(wbar[f], simpson ? G[f] : S[f], hds, coef, M);
    ++ctx->launches;
    CK(cudaGetLastError());
  }
  // getConc's mean subtraction of wA: its adjoint removes the mean of wAbar
  CKL(scft::launch_partial_sum<double>(wbar[0], M, M, B, ctx->partial, nblk, st));
  CKL(scft::launch_finalize_sum(ctx->partial, nblk, B, 1.0, sum, st));
  CKL(scft::launch_minus_average(wbar[0], sum, M, B, st));
  if (h_wabar) CK(cudaMemcpyAsync(h_wabar, wbar[0], dbytes, cudaMemcpyDeviceToHost, st));
  if (h_wbbar) CK(cudaMemcpyAsync(h_wbbar, wbar[1], dbytes, cudaMemcpyDeviceToHost, st));
  RC(scft_internal_sync_check(ctx));
  if (want_L) {
    for (int b = 0; b < B; ++b) {
      for (int a = 0; a < 3; ++a) h_Lbar[3 * b + a] = 0.0;
      auto S = [&](int kind) { return sums_h[(size_t)kind * B + b]; };
      for (int pi = 0; pi < np; ++pi)
        h_Lbar[3 * b + ctx->pass_axis[pi]] =
            S(ACC_L1 + pi) + S(ACC_L2 + pi) + qtot[b] / (double)M * S(ACC_Q + pi);
      for (int a = 0; a < 3; ++a)
        if (ctx->unit_c[a] != 0.0)
          h_Lbar[3 * b + a] =
              ctx->unit_c[a] * (S(ACC_U1) + S(ACC_U2) + qtot[b] / (double)M * S(ACC_UQ));
    }
  }
  return SCFT_OK;
}

// Box stress from the propagators stored by the last getConc (200 steps, ms: 128 x
// 128 x 64 pairs 22.2 -> 10.2, FP64 24 x 32 x 32 0.81 -> 0.50): for every contour step s
// (all independent, so batched `chunk` steps per launch) and axis a, W^-1 D_a W q+(s)
// contracted with q(s) in FP64, or (whole_axis) W K D_a W q(s-1) with q+(s).
template <typename R>
int stress_sums(scft_ctx *ctx, bool wide, double *acc) {
  AdjointState &A = *ctx->adj;
  const long long M = ctx->M;
  const int B = ctx->batch, nblk = kDotBlocks, np = (int)ctx->passes.size();
  cudaStream_t st = ctx->st;
  const int chunk = A.chunk;
  R *t[3];
  for (int k = 0; k < 3; ++k) t[k] = static_cast<R *>(A.smem) + (long long)k * chunk * M;
  R *winv = t[2] + (long long)chunk * M;
  CK(cudaMemsetAsync(acc, 0, sizeof(double) * 4 * B * nblk, st));
  struct Block { int q, qc, f, ns; };
  const Block blocks[2] = {{SCFT_Q_A, SCFT_Q_CA, 0, ctx->NsA}, {SCFT_Q_B, SCFT_Q_CB, 1, ctx->dNsB}};
  bool has_unit = false;
  for (int a = 0; a < 3; ++a) has_unit |= ctx->unit_c[a] != 0.0;
  bool quotient = false;
  for (int pi = 0; pi < np; ++pi) quotient |= !whole_axis(ctx, pi, wide);
  auto dots = [&](const DotArgs<R> &d, const R *y, int cnt) {
    const long long n = cnt * M;
    switch (d.n) {
      case 1: k_dots<R, 1, 4><<<nblk, kT, 0, st>>>(d, y, n); break;
      case 2: k_dots<R, 2, 2><<<nblk, kT, 0, st>>>(d, y, n); break;
      case 3: k_dots<R, 3, 2><<<nblk, kT, 0, st>>>(d, y, n); break;
      default: k_dots<R, 4, 1><<<nblk, kT, 0, st>>>(d, y, n); break;
    }
    ++ctx->launches;
    return cudaGetLastError();
  };
  for (const Block &bl : blocks) {
    const R *q = static_cast<const R *>(ctx->q[bl.q]);
    const R *qc = static_cast<const R *>(ctx->q[bl.qc]);
    const long long qbs = (long long)(bl.ns + 1) * M;
    for (int b = 0; b < B && bl.ns > 0; ++b) {
      const R *W = static_cast<const R *>(ctx->W[bl.f]) + b * M;
      if (quotient) {
        k_inverse<R><<<grid_for(M), kT, 0, st>>>(W, winv, M);
        ++ctx->launches;
        CK(cudaGetLastError());
      }
      auto slots = [&](int kind) { return acc + ((size_t)kind * B + b) * nblk; };
      for (int s1st = 1; s1st <= bl.ns; s1st += chunk) {
        const int cnt = std::min(chunk, bl.ns - s1st + 1);
        const R *qin = q + b * qbs + (long long)(s1st - 1) * M;    // q(s-1)
        const R *qcs = qc + b * qbs + (long long)s1st * M;         // q+(s)
        // the whole operators one after the other, then the quotient forms, which
        // keep a buffer each, with one reading of q(s)
        for (int pi = 0; pi < np; ++pi) {
          if (!whole_axis(ctx, pi, wide)) continue;
          DotArgs<R> one = {};
          RC(whole_term<R>(ctx, pi, qin, M, W, 0, cnt, t[0], t[1], t[2], st));
          one.x[0] = t[0];
          one.acc[0] = slots(pi);
          one.n = 1;
          CK(dots(one, qcs, cnt));
        }
        DotArgs<R> d = {};
        for (int pi = 0; pi < np; ++pi) {
          if (whole_axis(ctx, pi, wide)) continue;
          RC(scft_internal_deriv(ctx, pi, qcs, M, t[pi], M, W, winv, 0, cnt, st));
          d.x[d.n] = t[pi];
          d.acc[d.n++] = slots(pi);
        }
        if (has_unit) {   // <q+(s), W K W q(s-1)>
          d.x[d.n] = qcs;
          d.acc[d.n++] = slots(3);
        }
        if (d.n) CK(dots(d, qin + M, cnt));
      }
    }
  }
  return SCFT_OK;
}

template <typename R>
int stress_impl(scft_ctx *ctx, double *h_out) {
  AdjointState &A = *ctx->adj;
  const long long M = ctx->M;
  const int B = ctx->batch, nblk = kDotBlocks, np = (int)ctx->passes.size();
  cudaStream_t st = ctx->st;
  // [4 kinds][B][nblk]: passes 0..2 and the unit term, then [4][B] sums, a flag
  double *acc = reinterpret_cast<double *>(static_cast<unsigned char *>(A.smem) + A.sacc_off);
  double *sums = acc + (size_t)4 * B * nblk;
  int *flag = reinterpret_cast<int *>(sums + 4 * B);
  std::vector<double> s_h(4 * (size_t)B), hQ(B);
  int wide = 0;
  const R *const W[2] = {static_cast<const R *>(ctx->W[0]), static_cast<const R *>(ctx->W[1])};
  RC(whole_wanted<R>(ctx, W, flag, &wide));
  RC(stress_sums<R>(ctx, wide != 0, acc));
  k_sum_slots<<<4 * B, kT, 0, st>>>(acc, nblk, sums);
  ++ctx->launches;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(s_h.data(), sums, 8 * 4 * B, cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(hQ.data(), ctx->Q, 8 * B, cudaMemcpyDeviceToHost, st));
  RC(scft_internal_sync_check(ctx));
  for (int b = 0; b < B; ++b) {
    const double scale = -1.0 / ((double)M * hQ[b]);   // -d ln Q / dL
    for (int a = 0; a < 3; ++a) h_out[3 * b + a] = 0.0;
    for (int pi = 0; pi < np; ++pi)
      h_out[3 * b + ctx->pass_axis[pi]] = scale * s_h[(size_t)pi * B + b];
    for (int a = 0; a < 3; ++a)
      if (ctx->unit_c[a] != 0.0) h_out[3 * b + a] = scale * ctx->unit_c[a] * s_h[(size_t)3 * B + b];
  }
  return SCFT_OK;
}

}  // namespace

extern "C" {

int scft_adjoint(scft_ctx *ctx, const double *pha_bar, const double *phb_bar,
                 const double *Q_bar, double *wa_bar, double *wb_bar, double *L_bar,
                 int checkpoint_every) {
  if (!ctx) return SCFT_ERR_INVALID_ARG;
  const int N = ctx->NsA + ctx->dNsB;
  if (N < 1) return scft_fail(ctx, SCFT_ERR_UNSUPPORTED, "adjoint needs at least one step");
  if (checkpoint_every < 0) return scft_fail(ctx, SCFT_ERR_INVALID_ARG, "bad checkpoint interval");
  NvtxRange range("scft adjoint");
  int K = checkpoint_every ? checkpoint_every : (int)ceil(sqrt((double)N));
  if (K > N) K = N;
  CK(cudaSetDevice(ctx->p.device));
  RC(ensure_adjoint(ctx, K));
  return with_real(ctx, [&](auto r) {
    return adjoint_impl<decltype(r)>(ctx, pha_bar, phb_bar, Q_bar, wa_bar, wb_bar, L_bar);
  });
}

int scft_adjoint_checkpoints(scft_ctx *ctx, int checkpoint_every, int *slices,
                             long long *bytes) {
  if (!ctx || !slices) return SCFT_ERR_INVALID_ARG;
  const int N = ctx->NsA + ctx->dNsB;
  int K = checkpoint_every > 0 ? checkpoint_every : (int)ceil(sqrt((double)(N > 0 ? N : 1)));
  if (K > N) K = N > 0 ? N : 1;
  const int nck = (N + K - 1) / K + 1;
  *slices = 2 * nck + K + 1;   // both chains' checkpoints + one recompute segment
  if (bytes) *bytes = (long long)(*slices) * ctx->M * ctx->batch * ctx->rbytes;
  return SCFT_OK;
}

int scft_stress(scft_ctx *ctx, double *dF_dL) {
  if (!ctx || !dF_dL) return SCFT_ERR_INVALID_ARG;
  if (!ctx->have_conc)
    return scft_fail(ctx, SCFT_ERR_INVALID_ARG,
                     "no getConc at the current box: call scft_get_conc first");
  CK(cudaSetDevice(ctx->p.device));
  NvtxRange range("scft stress");
  if (!ctx->adj) ctx->adj = new AdjointState();
  AdjointState &A = *ctx->adj;
  if (!A.smem) {
    // up to 64 contour steps per launch.  FFT passes: the three chunk buffers <= 96
    // MB, with the slices that they are made from and contracted with in the L2.
    // Tensor-core passes, one CTA an SM, want long launches (128 x 128 x 64 FP64: 32
    // steps a launch 24 ms, 4 steps 32 ms): <= 768 MB.
    const long long per = ctx->M * ctx->rbytes;
    bool tc = false;
    for (const scft::AxisPlan &ap : ctx->passes) tc |= ap.tc != nullptr;
    int chunk = (int)std::min<long long>(64, std::max<long long>(1, ((tc ? 256LL : 32LL) << 20) / per));
    chunk = std::min(chunk, std::max(ctx->NsA, ctx->dNsB));
    chunk = std::max(chunk, 1);
    A.chunk = chunk;
    A.sacc_off = ((size_t)(3 * chunk + 1) * per + 255) & ~(size_t)255;
    A.sbytes = A.sacc_off + 8 * ((size_t)4 * ctx->batch * kDotBlocks + 4 * ctx->batch + 1);
    CK(cudaMalloc(&A.smem, A.sbytes));
  }
  return with_real(ctx, [&](auto r) { return stress_impl<decltype(r)>(ctx, dF_dL); });
}

int scft_relax_cell(scft_ctx *ctx, int axes_mask, double tol_w, double tol_stress,
                    int max_outer, int max_inner, double step0, int *outer_iters,
                    double *dF_dL, double *out5) {
  if (!ctx || !(tol_w > 0) || !(tol_stress > 0) || max_outer < 1 || max_inner < 1 ||
      !(step0 > 0) || (axes_mask & ~7) || !axes_mask)
    return SCFT_ERR_INVALID_ARG;
  if (ctx->batch != 1)
    return scft_fail(ctx, SCFT_ERR_UNSUPPORTED, "cell relaxation needs batch == 1 (one box)");
  double L[3] = {ctx->p.lx, ctx->p.ly, ctx->p.lz}, sig[3], fe[5];
  double L_prev[3] = {0, 0, 0}, sig_prev[3] = {0, 0, 0};
  double alpha = step0;
  // Inexact inner solves: far from the stress-free box the fields need not be
  // converged tightly, so each round converges to max(tol_w, stress/10) of
  // the previous round (at most 1e-3); the last round always reaches tol_w.
  double tol = std::max(tol_w, 1e-3);
  int it = 0;
  for (;;) {
    int iters = 0;
    RC(scft_converge(ctx, tol, max_inner, &iters, fe));
    RC(scft_internal_get_conc(ctx));   // propagators of the converged fields
    RC(scft_stress(ctx, sig));
    double smax = 0.0;
    for (int a = 0; a < 3; ++a)
      if (axes_mask >> a & 1) smax = std::max(smax, fabs(sig[a]));
    ++it;
    if (it >= max_outer) break;
    if (smax < tol_stress) {
      if (tol <= tol_w) break;
      tol = tol_w;   // stress-free at a loose tolerance: tighten, same box
      continue;
    }
    tol = std::max(tol_w, std::min(1e-3, 0.1 * smax));
    // Barzilai-Borwein step on F*(L), whose gradient is the stress
    if (it > 1) {
      double ss = 0.0, sy = 0.0;
      for (int a = 0; a < 3; ++a)
        if (axes_mask >> a & 1) {
          const double dl = L[a] - L_prev[a], dg = sig[a] - sig_prev[a];
          ss += dl * dl;
          sy += dl * dg;
        }
      if (sy > 0.0) alpha = ss / sy;
    }
    double Ln[3] = {L[0], L[1], L[2]};
    for (int a = 0; a < 3; ++a) {
      if (!(axes_mask >> a & 1)) continue;
      double d = -alpha * sig[a];
      const double cap = 0.05 * L[a];   // at most 5% per step
      d = std::max(-cap, std::min(cap, d));
      Ln[a] = L[a] + d;
    }
    for (int a = 0; a < 3; ++a) {
      L_prev[a] = L[a];
      sig_prev[a] = sig[a];
      L[a] = Ln[a];
    }
    RC(scft_set_box(ctx, L[0], L[1], L[2]));
  }
  if (outer_iters) *outer_iters = it;
  if (dF_dL) for (int a = 0; a < 3; ++a) dF_dL[a] = sig[a];
  if (out5) for (int k = 0; k < 5; ++k) out5[k] = fe[k];
  return SCFT_OK;
}

}  // extern "C"
