// Host-side launchers of the SCFT kernels (all run on one CUDA stream each).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "dfloat.cuh"

namespace scft {

// One per-axis pass of the separable diffusion operator exp(-k^2 ds):
// every line along the axis is transformed, multiplied by the real, even
// gain g[k] (= exp(-ds*k^2)/N, the reference's kxyzdz factor split per axis),
// and transformed back.  Two real lines are packed as the real and imaginary
// parts of one complex line; because g is real and even the two lines do not
// mix.  Geometry of the real lines of one instance:
//   element (outer o, real line r, position n) at  o*s_outer + r*s_pair + n*s_n
struct AxisPlan {
  int n;                 // line length
  int nfac;              // radix plan (Stockham stages), product == n
  int fac[24];
  long long s_n, s_pair, s_outer;
  int n_real;            // real lines per outer group (paired 2 by 2)
  int n_outer;           // outer groups per instance
  int n_fast;            // 1: consecutive threads walk n (contiguous lines)
  int flat_nx;           // column passes: 0, or the row length when the columns run over a
                         // flattened (row, outer) index: column c sits at
                         // (c / flat_nx) * s_outer + c % flat_nx (n_outer 1)
  int tl;                // complex lines per CTA tile
  int use_fast;          // FP32 register-resident kernel (k_fast.cu) handles this pass
  const void *twiddle;   // device: n complex, exp(-2*pi*i*m/n), working precision
  const void *gain;      // device: n reals, working precision
  const void *tc;        // device: the gain's tensor-core table (k_tc.cu), or null
};

// One pass over up to kMaxSet independent propagators at once (the lockstep
// march chains): set k reads in[k] (+ b*in_bs), multiplies by pre[k], filters,
// multiplies by post[k] and writes out[k] (+ b*out_bs), for every instance b.
constexpr int kMaxSet = 2, kStepSet = 3;
// One line set of a batched pass over several contexts (a group's lockstep
// march, FP32): the set's buffers (one instance each) and gain tables.
struct PassDesc {
  const float *in;
  float *out;
  const float *pre, *post;   // Boltzmann factor on load / on store, or null
  const float *gain;         // the set's gain table of this pass's axis (x for a plane pass)
  const float *gain_y;       // x+y plane passes: the y axis's gain table
  const void *tc, *tc_y;     // the set's tensor-core tables (tc_y: plane passes)
};
// (NS: sets it has room for; kStepSet only in scft_internal_steps, since the
// longer arguments cost every launch about 1 % of a small pass)
template <typename R, int NS = kMaxSet> struct PassSet {
  const R *in[NS];
  R *out[NS];
  const R *pre[NS];
  const R *post[NS];
  long long in_bs[NS], out_bs[NS];
  long long w_bs;
  int nset;
  int batch;
  unsigned *err;   // device error word (bounded-wait timeouts), may be null for non-pipelined kernels
  // fused step pairs only (launch_zz / launch_xyxy): where the finished
  // propagator slice goes; `out` then receives the next step's intermediate
  R *qout[NS];
  long long qout_bs[NS];
  // FP32 per-axis and x+y plane passes: when set, line set blockIdx.z takes
  // its buffers and gains from desc[blockIdx.z] (nset 1, batch = sets)
  const PassDesc *desc;
};

#ifdef __CUDACC__
// The line set of a CTA (blockIdx.z = set * batch + instance), and its entry of
// one of the set's arrays: selected, not indexed, which is a load behind a load.
template <typename R, int NS>
__device__ __forceinline__ int set_of(const PassSet<R, NS> &ps) {
  const int z = blockIdx.z;
  if (NS == 2) return z >= ps.batch ? 1 : 0;
  return z < ps.batch ? 0 : (z < 2 * ps.batch ? 1 : 2);
}
template <typename V> __device__ __forceinline__ V of_set(const V (&a)[2], int set) {
  return set ? a[1] : a[0];
}
template <typename V> __device__ __forceinline__ V of_set(const V (&a)[3], int set) {
  return set == 0 ? a[0] : (set == 1 ? a[1] : a[2]);
}
#endif
// The first sets of a set for more, or the other way round (as many as fit).
template <int NS, typename R, int MS> PassSet<R, NS> with_sets(const PassSet<R, MS> &a, int first = 0) {
  PassSet<R, NS> p = {};
  for (int k = 0; k < NS && first + k < MS; ++k) {
    p.in[k] = a.in[first + k];
    p.out[k] = a.out[first + k];
    p.pre[k] = a.pre[first + k];
    p.post[k] = a.post[first + k];
    p.in_bs[k] = a.in_bs[first + k];
    p.out_bs[k] = a.out_bs[first + k];
    p.qout[k] = a.qout[first + k];
    p.qout_bs[k] = a.qout_bs[first + k];
  }
  p.nset = a.nset - first < NS ? a.nset - first : NS;
  p.w_bs = a.w_bs;
  p.batch = a.batch;
  p.err = a.err;
  p.desc = a.desc;
  return p;
}

// Register-resident pass (k_fast.cu): n in {32, 64, 128, 256} (FP32) or
// {32, 64, 128} (FP64), and n_real a multiple of 64.
bool fast_line_supported(const AxisPlan &ap, size_t real_bytes = 4);
// Fused x+y pass over whole z-planes (k_fast.cu): Nx, Ny in {64, 128}.
bool xy_fusable(const AxisPlan &apx, const AxisPlan &apy);
template <int NS>
cudaError_t launch_xy(const AxisPlan &apx, const AxisPlan &apy, const PassSet<float, NS> &ps,
                      cudaStream_t st);
cudaError_t fast_line_prepare();
// x+y passes of 256 x 256 planes (k_plane256.cu): a cluster of two CTAs per
// plane, the y lines read across the pair through distributed shared memory;
// launch_xy / launch_xyxy dispatch here for such planes.
bool plane256_fusable(const AxisPlan &apx, const AxisPlan &apy);
cudaError_t plane256_prepare();
cudaError_t launch_xy256(const AxisPlan &apx, const AxisPlan &apy, const PassSet<float> &ps,
                         cudaStream_t st);
cudaError_t launch_xyxy256(const AxisPlan &apx, const AxisPlan &apy, const PassSet<float> &ps,
                           cudaStream_t st);
// bounded-wait self-test: sets bit 4 of *err after `limit` clocks
cudaError_t launch_wait_selftest(unsigned *err, long long limit, cudaStream_t st);
template <typename R, int NS>
cudaError_t launch_fast_line(const AxisPlan &ap, const PassSet<R, NS> &ps, cudaStream_t st);
// Fused step pairs.  The axis filters commute, so consecutive contour steps
// can run their passes in alternating order (x+y then z, z then x+y); the
// end of one step and the start of the next are then the same pass type and
// run as one kernel: qout = post * K_a(in), out = K_a(post * qout), with
// K_a the z filter (launch_zz) or the x+y filters (launch_xyxy).
cudaError_t launch_zz(const AxisPlan &ap, const PassSet<float> &ps, cudaStream_t st);
cudaError_t launch_zz(const AxisPlan &ap, const PassSet<double> &ps, cudaStream_t st);
cudaError_t launch_zz(const AxisPlan &ap, const PassSet<dfloat> &ps, cudaStream_t st);
// the same on x lines (rows contiguous), for grids without the x+y plane
cudaError_t launch_xx(const AxisPlan &ap, const PassSet<float> &ps, cudaStream_t st);
cudaError_t launch_xx(const AxisPlan &ap, const PassSet<double> &ps, cudaStream_t st);
cudaError_t launch_xx(const AxisPlan &ap, const PassSet<dfloat> &ps, cudaStream_t st);
cudaError_t launch_xyxy(const AxisPlan &apx, const AxisPlan &apy, const PassSet<float> &ps,
                        cudaStream_t st);

// Tensor-core line filter (k_tc.cu): exact integer convolution of lines of any
// even length, up to 128 points (FP64: 7 digits) or 224 (FP32: 4 digits).  pair (FP32): a fused step pair (qout = post * K(in),
// out = K(post * qout)).
bool tc_line_possible(int n, int nd);
bool tc_line_usable(int n, int nd);   // on this device, after tc_prepare
long long tc_pass_ctas(const AxisPlan &ap, int nd);
bool tc_planes_wanted(int nx, int ny, int nz, int nd, int batch);
size_t tc_table_bytes(int n, int nd);
bool tc_build_table(const double *gain, int n, int nd, std::vector<unsigned char> &table,
                    double *row_sum);
cudaError_t tc_prepare();
cudaError_t launch_tc(const AxisPlan &ap, const PassSet<float, kStepSet> &ps, bool pair,
                      cudaStream_t st);
cudaError_t launch_tc(const AxisPlan &ap, const PassSet<double, kStepSet> &ps, bool pair,
                      cudaStream_t st);
// One pass of the fused FP64 march, whose intermediates are 64-bit integers (batch
// instances; strides in elements): a point's value is its integer times 2^u, u that of
// the line that the pass before filtered it in.
struct FixPass {
  const void *in;            // FIRST: FP64, else integers
  void *out;                 // integers (not LAST)
  void *q;                   // PAIR, LAST: the finished slice
  const double *w;           // the factors
  const int16_t *u_in;       // units by lines of the pass before ...
  int16_t *u_out;            // ... and of this one, in the order of their offsets
  // point k of line c: (c / u_div) * u_quo + (c % u_div) * u_rem + k * u_step
  int u_div, u_quo, u_rem, u_step;
  long long in_bs, out_bs, q_bs, w_bs, u_in_bs, u_out_bs;
  int batch;
  unsigned *err;             // device error word (bounded-wait timeouts)
};
constexpr int kFixFirst = 0, kFixMid = 1, kFixPair = 2, kFixLast = 3;
cudaError_t launch_fix(const AxisPlan &ap, int mode, const FixPass &fp, cudaStream_t st);
// Both axes of whole planes in one launch: x, y, the factor (q stored), the
// factor, y, x (without qout, or batched: pre, x, y); FP64 also a film's whole march
// segment.
cudaError_t launch_planes(const AxisPlan &apx, const AxisPlan &apy,
                          const PassSet<float, kStepSet> &ps, cudaStream_t st);
cudaError_t launch_planes(const AxisPlan &apx, const AxisPlan &apy, const FixPass &fp, int steps,
                          long long q_step, cudaStream_t st);

// Generic mixed-radix Stockham line filter (any n whose prime factors are
// <= 61).  in/out may not alias.  pre multiplies the input, post the output
// (elementwise, indexed like one instance's grid); either may be null.
template <typename R>
cudaError_t launch_line_filter(const AxisPlan &ap, const R *in, long long in_bstride, R *out,
                               long long out_bstride, const R *pre, const R *post,
                               long long w_bstride, int batch, cudaStream_t st);
// The same over n line sets described by desc[0..n) (FP32, device memory).
cudaError_t launch_line_filter_desc(const AxisPlan &ap, const PassDesc *desc, int n,
                                    cudaStream_t st);

size_t line_filter_smem_bytes(const AxisPlan &ap, size_t real_bytes);
constexpr int kLineSmemMax = 200 * 1024;
cudaError_t line_filter_prepare();

// ---- residual and Anderson mixing (k_anderson.cu) ----
int anderson_max_slots();
// residual of phi_w's update (err[b][2] = max, rms); optionally stores
// u = w + lam_u d and d into a history slot (hu, hd: [b][2][M] double-float
// pairs), copies w to wprev ([b][2][M] FP64) and/or applies the simple step
// w += wopt*d (4 kernels)
cudaError_t launch_residual(double *wa, double *wb, const double *pha, const double *phb,
                            double hAB, double wcmp, double wopt, long long M, int batch,
                            void *hu, void *hd, double lam_u, double *wprev, double *partial,
                            int nblk, double *err, cudaStream_t st);
// Gram row <d_c, d_j> (double-float ring slots) into the FP64 ring matrix
// (2 kernels)
cudaError_t launch_gram_row(const void *dc, const void *const *dj, const int *slots, int n,
                            int c, int m1, long long M, int batch, double *partial, int nblk,
                            double *G, cudaStream_t st);
// weights a[b][m1], step lam[b] and mode lam[batch + b] (1 Anderson, 0 simple)
cudaError_t launch_anderson_solve(const double *G, const double *err, int c, int hist, int m1,
                                  double start, double lambda, double wopt, int batch,
                                  double *a, double *lam, cudaStream_t st);
// The update w0 -> (wa, wb) without its component along the rigid shifts of
// w0 ([b][2][M], central differences, periodic): three kernels; partial holds
// batch*9*nblk doubles, alpha batch*3.
cudaError_t launch_remove_translation(double *wa, double *wb, const double *w0, int nx, int ny,
                                     int nz, int batch, double *partial, int nblk,
                                     double *alpha, cudaStream_t st);
// w_new = sum_k a_k u_k over the listed ring slots (Anderson step) or
// w + lam d_c (simple step), per instance as the solve decided
cudaError_t launch_anderson_update(double *wa, double *wb, const void *const *hu, const void *dc,
                                   const int *idx, int n, const double *a, const double *lam,
                                   int m1, long long M, int batch, cudaStream_t st);

// ---- field kernels (k_fields.cu) ----
// W = exp(-w*ds2) in precision R, for batch*M points (w is FP64).
template <typename R>
cudaError_t launch_boltzmann(const double *w, R *W, long long n, double ds2, cudaStream_t st);
template <typename R>
cudaError_t launch_fill(R *x, long long n, R v, long long bstride, int batch, cudaStream_t st);
// dst[b*dst_bstride + i] = src[b*src_bstride + i], i < M
template <typename R>
cudaError_t launch_copy_slice(R *dst, long long dst_bstride, const R *src, long long src_bstride,
                              long long M, int batch, cudaStream_t st);
template <typename R>
cudaError_t launch_cast_slice(double *dst, long long dst_bstride, const R *src,
                              long long src_bstride, long long M, int batch, cudaStream_t st);

// Deterministic per-instance sums: partial[b*nblk+k] then finalize.
int reduce_blocks(long long M);
template <typename R>
cudaError_t launch_partial_sum(const R *x, long long bstride, long long M, int batch,
                               double *partial, int nblk, cudaStream_t st);
cudaError_t launch_finalize_sum(const double *partial, int nblk, int batch, double scale,
                                double *out, cudaStream_t st);
// data -= sum/M  (minus_average)
cudaError_t launch_minus_average(double *data, const double *sum, long long M, int batch,
                                 cudaStream_t st);
// Q = sum/M ; ffl = ds0/Q  (cal_ql + host lines of getConc)
cudaError_t launch_q_ffl(const double *sum, long long M, double ds0, int batch, double *Q,
                         double *ffl, cudaStream_t st);
// Weight of contour point s (0..n) of a block of n steps: the reference's
// trapezoid (1/2 at both ends, 1 inside; the n == 0 block has the single
// weight 1/2, cuda_aid.cu:87-107), or Simpson (1/3 rule; for odd n >= 3 the
// 3/8 rule over the last three steps; n == 1 stays trapezoid).
double contour_weight(int s, int n, bool simpson);
// The same weights in kernel form: interior points 1..m-1 take c_odd (odd s)
// or c_even (even s); up to five listed points take their own weight.
struct ContourWeights {
  int m, nspec;
  double c_odd, c_even;
  int s[5];
  double w[5];
};
ContourWeights contour_weights(int n, bool simpson);
// phi = ffl * contour sum of q*qc with the weights above (w_to_phi_go)
template <typename R>
cudaError_t launch_contour_phi(const R *q, const R *qc, int ns, long long M, int batch,
                               const double *ffl, double *phi, bool simpson, cudaStream_t st);
// simple mixing (phi_w); writes the residual max-norm partials if resid != null
cudaError_t launch_phi_w(double *wa, double *wb, const double *pha, const double *phb,
                         double hAB, double wopt, double wcmp, long long M, int batch,
                         cudaStream_t st);
// propagator [b][s][M] -> g[b][r][s] FP64 (the reference's layout)
template <typename R>
cudaError_t launch_q_to_reference_layout(const R *q, int ns, long long M, int batch, double *g,
                                         cudaStream_t st);
// phi_w_constrained (ex == 0) / phi_w_constrainedEx (ex != 0)
cudaError_t launch_phi_w_constrained(double *wa, double *wb, const double *pha, const double *phb,
                                     const double *target, double hAB, double lambda, int ex,
                                     long long M, int batch, cudaStream_t st);
// free energy partials: sums of hAB*pa*pb, wa*pa+wb*pb and max|1-pa-pb|
cudaError_t launch_free_energy_partials(const double *wa, const double *wb, const double *pha,
                                        const double *phb, double hAB, long long M, int batch,
                                        double *partial, int nblk, cudaStream_t st);
cudaError_t launch_free_energy_finalize(const double *partial, int nblk, int batch, long long M,
                                        const double *Q, double *out5, cudaStream_t st);

}  // namespace scft
