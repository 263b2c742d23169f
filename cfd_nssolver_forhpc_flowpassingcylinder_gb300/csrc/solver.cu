// Pressure Poisson solvers on the 7-point Neumann operator.
//
// BiCGSTAB follows bicgstabRe2::solve (inc/solver/bicgstabRe2.hpp:84-180) step for step:
// warm start, relative-residual stop, rho restart, iteration cap and NaN recovery.  Every
// global dot product is a deterministic two-stage FP64 reduction (reduce.cuh) whose last
// block also makes the scalar decisions (alpha, omega, stop test, beta, restart), so no
// host round trip happens inside an iteration.  Every kernel returns at once when
// sc->done is set, which lets the host enqueue iterations in chunks (captured as CUDA
// graphs) and poll only between chunks.
//
// Launch geometry: 3-D blocks (bx along k, by along j) with the grid's z dimension
// striding over i, so each thread knows its (i, j, k) without a division.
//
// FP64 (the plain path, bound by the FP64 pipe): five kernels per iteration, no
// recomputation.  FP32 (inner solve of the mixed path, bound by HBM): three kernels per
// iteration; the p update is fused into the next SpMV and s into its SpMV by
// recomputing them at the stencil points (L1-resident), 17 instead of 19 words per cell.
#include <algorithm>
#include <atomic>

#include "cfdgb_internal.cuh"
#include "kernels.h"
#include "reduce.cuh"

namespace cfdgb {

// (ic, jc, kc) of this thread and the loop over the i planes it owns.
#define FOR_CELLS(g)                                               \
  const int kc = blockIdx.x * blockDim.x + threadIdx.x;            \
  const int jc = blockIdx.y * blockDim.y + threadIdx.y;            \
  const bool on_ = (kc < (g).nzc) && (jc < (g).nyc);               \
  for (int ic = blockIdx.z; on_ && ic < (g).nxc; ic += gridDim.z)

// the same, four planes of a thread's column in flight at once (short bodies that stream)
#define FOR_CELLS4(g)                                              \
  const int kc = blockIdx.x * blockDim.x + threadIdx.x;            \
  const int jc = blockIdx.y * blockDim.y + threadIdx.y;            \
  const bool on_ = (kc < (g).nzc) && (jc < (g).nyc);               \
  _Pragma("unroll 4") for (int ic = blockIdx.z; on_ && ic < (g).nxc; ic += gridDim.z)

#define ROW(g) ((((long long)ic * (g).nyc + jc) * (g).nzc) + kc)

__device__ __forceinline__ int cls_of(const Geo &g, int ic, int jc, int kc) { return row_class(g, ic, jc, kc); }

// y = (A f)(row) where f(q) is evaluated on demand at the stencil points
template <typename T, class F>
__device__ __forceinline__ T stencil_apply(const Geo &g, const Stencil<T> &st, int ic, int jc, int kc,
                                           long long row, F &&f, T &center) {
  const long long nyz = (long long)g.nyc * g.nzc;
  if constexpr (sizeof(T) == sizeof(double)) {
    if (g.nonuni) {  // stretched grid (FP64 solvers only): the rows stored per context
      const double *__restrict__ cs = g.cof[st.jac] + row;
      const long long n = g.ncell, zm = z_minus(g, kc, row), zp = z_plus(g, kc, row);
      T sum = T(0);
      if (ic > 0) sum += cs[0] * f(row - nyz);
      if (jc > 0) sum += cs[n] * f(row - g.nzc);
      if (zm >= 0) sum += cs[2 * n] * f(zm);
      center = f(row);
      sum += cs[3 * n] * center;
      if (zp >= 0) sum += cs[4 * n] * f(zp);
      if (jc < g.nyc - 1) sum += cs[5 * n] * f(row + g.nzc);
      if (ic < g.nxc - 1) sum += cs[6 * n] * f(row + nyz);
      return sum;
    }
  }
  const T *c = st.c[cls_of(g, ic, jc, kc)];
  const long long zm = z_minus(g, kc, row), zp = z_plus(g, kc, row);
  T sum = T(0);
  if (ic > 0) sum += c[0] * f(row - nyz);
  if (jc > 0) sum += c[1] * f(row - g.nzc);
  if (zm >= 0) sum += c[2] * f(zm);
  center = f(row);
  sum += c[3] * center;
  if (zp >= 0) sum += c[4] * f(zp);
  if (jc < g.nyc - 1) sum += c[5] * f(row + g.nzc);
  if (ic < g.nxc - 1) sum += c[6] * f(row + nyz);
  return sum;
}

// FP32 form of the same operator: every row sums to zero (Neumann rows: the diagonal is
// minus the sum of the neighbour coefficients), so A f = sum_nb c_nb (f_nb - f_centre).
// Differencing first makes A exactly singular on constants in FP32 and keeps the rounding
// error proportional to the local differences rather than to |f|: on the smooth modes that
// dominate late in a solve, the plain 7-term sum would lose ~eps32 * cond(A) (~1e-2 at
// 512 cells per axis) and stall the iteration there.
template <class F>
__device__ __forceinline__ float stencil_apply_diff(const Geo &g, const Stencil<float> &st, int ic, int jc, int kc,
                                                    long long row, F &&f, float &center) {
  const long long nyz = (long long)g.nyc * g.nzc;
  const long long zm = z_minus(g, kc, row), zp = z_plus(g, kc, row);
  const float fc = f(row);
  center = fc;
  float sum = 0.0f;
  if (g.nonuni) {  // stretched grid (MIXED): its rows stored in FP32, [7][ncell]
    const float *__restrict__ cs = g.cof32[st.jac] + row;
    const long long n = g.ncell;
    if (ic > 0) sum = fmaf(cs[0], f(row - nyz) - fc, sum);
    if (jc > 0) sum = fmaf(cs[n], f(row - g.nzc) - fc, sum);
    if (zm >= 0) sum = fmaf(cs[2 * n], f(zm) - fc, sum);
    if (zp >= 0) sum = fmaf(cs[4 * n], f(zp) - fc, sum);
    if (jc < g.nyc - 1) sum = fmaf(cs[5 * n], f(row + g.nzc) - fc, sum);
    if (ic < g.nxc - 1) sum = fmaf(cs[6 * n], f(row + nyz) - fc, sum);
    return sum;
  }
  const float *c = st.c[cls_of(g, ic, jc, kc)];
  if (ic > 0) sum = fmaf(c[0], f(row - nyz) - fc, sum);
  if (jc > 0) sum = fmaf(c[1], f(row - g.nzc) - fc, sum);
  if (zm >= 0) sum = fmaf(c[2], f(zm) - fc, sum);
  if (zp >= 0) sum = fmaf(c[4], f(zp) - fc, sum);
  if (jc < g.nyc - 1) sum = fmaf(c[5], f(row + g.nzc) - fc, sum);
  if (ic < g.nxc - 1) sum = fmaf(c[6], f(row + nyz) - fc, sum);
  return sum;
}

// b - (A x)(row) as one FMA chain from b, the terms in stencil_apply's order (the MIXED
// refinement's residual: FP64-pipe-bound, so the subtraction folds into the chain)
__device__ __forceinline__ double resid_at(const Geo &g, const Stencil<double> &st, const double *__restrict__ x, int ic,
                                          int jc, int kc, long long row, double bb) {
  const long long nyz = (long long)g.nyc * g.nzc;
  const long long zm = z_minus(g, kc, row), zp = z_plus(g, kc, row);
  double r = bb;
  if (g.nonuni) {  // stretched grid: the rows stored per context
    const double *__restrict__ cs = g.cof[st.jac] + row;
    const long long n = g.ncell;
    if (ic > 0) r = fma(-cs[0], x[row - nyz], r);
    if (jc > 0) r = fma(-cs[n], x[row - g.nzc], r);
    if (zm >= 0) r = fma(-cs[2 * n], x[zm], r);
    r = fma(-cs[3 * n], x[row], r);
    if (zp >= 0) r = fma(-cs[4 * n], x[zp], r);
    if (jc < g.nyc - 1) r = fma(-cs[5 * n], x[row + g.nzc], r);
    if (ic < g.nxc - 1) r = fma(-cs[6 * n], x[row + nyz], r);
    return r;
  }
  const double *c = st.c[cls_of(g, ic, jc, kc)];
  if (ic > 0) r = fma(-c[0], x[row - nyz], r);
  if (jc > 0) r = fma(-c[1], x[row - g.nzc], r);
  if (zm >= 0) r = fma(-c[2], x[zm], r);
  r = fma(-c[3], x[row], r);
  if (zp >= 0) r = fma(-c[4], x[zp], r);
  if (jc < g.nyc - 1) r = fma(-c[5], x[row + g.nzc], r);
  if (ic < g.nxc - 1) r = fma(-c[6], x[row + nyz], r);
  return r;
}

template <typename T>
__device__ __forceinline__ T spmv_at(const Geo &g, const Stencil<T> &st, const T *__restrict__ x, int ic, int jc,
                                     int kc, long long row) {
  T c;
  return stencil_apply<T>(g, st, ic, jc, kc, row, [&](long long q) { return x[q]; }, c);
}

// ---- FP64 set-up: bicgstabRe2.hpp:86-106 ----
// restart: 1 for the preconditioned iteration, whose first p kernel then takes p = r0 = r1
__global__ void __launch_bounds__(kBlock) k_bicg_setup64(Geo g, Stencil<double> st, KrylovVecs<double> v,
                                                          const double *__restrict__ b, double *px1, double *px2,
                                                          double *part, SolverScal *sc, int restart) {
  double acc[2] = {0.0, 0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double bb = b[row];
    const double r = bb - spmv_at<double>(g, st, v.x, ic, jc, kc, row);
    v.r0[row] = r;
    v.r1[row] = r;
    v.p1[row] = r;
    px2[row] = px1[row];
    px1[row] = v.x[row];
    acc[0] += bb * bb;
    acc[1] += r * r;
  }
  double out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[0], out) && lin_tid() == 0) {
    sc->timestep += 1;
    sc->norm0 = sqrt(out[0]);
    sc->rho = out[1];
    sc->iter = 0;
    sc->done = 0;
    sc->status = 0;
    sc->fault = 0;
    sc->restart = restart;
    sc->relres = 0.0;
  }
}

// ---- FP64 iteration: five kernels ----
// K1: ap = A p1, alpha = rho / <ap, r0>
__global__ void __launch_bounds__(kBlock) k64_ap(Geo g, Stencil<double> st, KrylovVecs<double> v, double *part,
                                                 SolverScal *sc) {
  if (sc->done) return;
  double a[1] = {0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double y = spmv_at<double>(g, st, v.p1, ic, jc, kc, row);
    v.ap[row] = y;
    a[0] += y * v.r0[row];
  }
  double out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}

// K2: s = r1 - alpha ap
__global__ void __launch_bounds__(kBlock) k64_s(Geo g, KrylovVecs<double> v, const SolverScal *sc) {
  if (sc->done) return;
  const double a = sc->alpha;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    v.s[row] = v.r1[row] - a * v.ap[row];
  }
}

// K3: as = A s, omega = <as, s> / <as, as>
__global__ void __launch_bounds__(kBlock) k64_as(Geo g, Stencil<double> st, KrylovVecs<double> v, double *part,
                                                 SolverScal *sc) {
  if (sc->done) return;
  double a[2] = {0.0, 0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double y = spmv_at<double>(g, st, v.s, ic, jc, kc, row);
    v.as[row] = y;
    a[0] += y * v.s[row];
    a[1] += y * y;
  }
  double out[2];
  if (grid_sum<2>(a, part, &sc->cnt[2], out) && lin_tid() == 0) sc->omega = out[0] / out[1];
}

// The scalar work that ends an iteration is one thread's chain of FP64 divisions, each a
// few dozen instructions at 64 cycles: warp 0 of the last block takes them on three lanes
// at once (one division sequence instead of three).  a0 / b0, a1 / b1, a2 / b2 in every lane
// of the warp.
__device__ __forceinline__ void div3(double a0, double b0, double a1, double b1, double a2, double b2, double &q0,
                                     double &q1, double &q2) {
  const int l = lin_tid() & 31;
  const double q = (l == 0 ? a0 : l == 1 ? a1 : a2) / (l == 0 ? b0 : l == 1 ? b1 : b2);
  q0 = __shfl_sync(0xffffffffu, q, 0);
  q1 = __shfl_sync(0xffffffffu, q, 1);
  q2 = __shfl_sync(0xffffffffu, q, 2);
}

// stop test, beta and restart decision of bicgstabRe2.hpp:128-176 (last block, warp 0);
// n2 = ||r1||^2, rr = <r1, r0>.  Every scalar is loaded before the decisions, so that their
// latencies overlap.
template <bool FP32>
__device__ __forceinline__ void finish_iteration(SolverScal *sc, double n2, double rr) {
  if (lin_tid() >= 32) return;
  const double tol = sc->tol, rho_old = sc->rho, rn = sqrt(n2);
  const double peak_max = sc->rmax, rstart = sc->rstart, delta = sc->delta, peak = sc->peak, best = sc->best,
               snap_rel = sc->snap_rel, thr = sc->restart_thr;
  const int iter = sc->iter, maxit = sc->maxit, timestep = sc->timestep, snap_iter = sc->snap_iter,
            stall = sc->stall;
  const double omega = sc->omega;
  double relres, ao, rq;
  div3(rn, sc->norm0, sc->alpha, omega, rr, rho_old, relres, ao, rq);
  const double beta = ao * rq;
  if (lin_tid() != 0) return;
  sc->relres = relres;
  if (FP32) {
    // MIXED sweep: hand over to the FP64 refinement once the residual has dropped by delta
    // below the sweep's start, or by peak below the sweep's largest one (BiCGSTAB's
    // residual can rise far above its start before it falls, and an FP32 recursion cannot
    // follow it down many decades below such a peak), or looks converged
    if (relres < best) sc->best = relres;
    // keep this iterate (the next x update copies it) once its residual has halved since
    // the last one kept: a few copies per sweep, and the sweep's correction is never worse
    // than that kept iterate, whatever the residual does afterwards
    const bool snap = relres <= 0.5 * snap_rel;
    sc->snap = snap;
    if (snap) {
      sc->snap_rel = relres;
      sc->snap_iter = iter;
    }
    if (!isfinite(relres)) {
      sc->done = 1;
      sc->status = CFDGB_ENAN;
    } else if (iter > 16 && relres > 1e3 * (relres < best ? relres : best)) {
      // runaway growth (BiCGSTAB's ordinary bumps stay far below this)
      sc->done = 1;
      sc->status = CFDGB_ENOCONV;
    } else if (iter >= maxit) {
      sc->done = 1;
      sc->status = CFDGB_ENOCONV;
      sc->iter = iter + 1;
    } else if (relres < tol || rn < delta * rstart || rn < peak * peak_max) {
      sc->done = 1;
      sc->status = kStatusRefine;
      sc->iter = iter + 1;
    } else if (!snap && iter - snap_iter >= stall) {
      sc->done = 1;
      sc->status = CFDGB_ENOCONV;
      sc->iter = iter + 1;
    } else {
      sc->beta = beta;
      const bool broke = !(isfinite(beta) && omega != 0.0 && rr != 0.0);  // Lanczos breakdown
      sc->restart = broke ? 1 : 0;
      sc->rho = broke ? n2 : rr;
      sc->rmax = fmax(peak_max, rn);
      sc->iter = iter + 1;
    }
    return;
  }
  if (relres < tol) {  // :129
    sc->done = 1;
  } else if (iter >= maxit) {  // :133
    sc->done = 1;
    sc->status = CFDGB_ENOCONV;
  } else {  // :156-176
    sc->rho = rr;
    sc->beta = beta;
    sc->restart = !(timestep < 10 || fabs(rho_old) > thr);
    sc->iter = iter + 1;
  }
}

// K4: x += alpha p1 + omega s; r1 = s - omega as; ||r1||^2, <r1, r0>
__global__ void __launch_bounds__(kBlock) k64_xr(Geo g, KrylovVecs<double> v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const double a = sc->alpha, w = sc->omega;
  double acc[2] = {0.0, 0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double s = v.s[row];
    v.x[row] = fma(w, s, fma(a, v.p1[row], v.x[row]));  // two FP64 ops instead of three
    const double r1 = fma(-w, v.as[row], s);
    v.r1[row] = r1;
    acc[0] += r1 * r1;
    acc[1] += r1 * v.r0[row];
  }
  double out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[3], out)) finish_iteration<false>(sc, out[0], out[1]);
}

// K5: p1 = r1 + beta (p1 - omega ap), or restart r0 = p1 = r1
__global__ void __launch_bounds__(kBlock) k64_p(Geo g, KrylovVecs<double> v, const SolverScal *sc) {
  if (sc->done) return;
  const double b = sc->beta, w = sc->omega;
  const bool rst = sc->restart != 0;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double r1 = v.r1[row];
    if (rst) {
      v.r0[row] = r1;
      v.p1[row] = r1;
    } else {
      v.p1[row] = r1 + b * (v.p1[row] - w * v.ap[row]);
    }
  }
}

// ---- FP32 iteration: three fused kernels; p and ap are double-buffered by parity ----
struct Vec32 {
  float *x, *r0, *r1, *s, *as, *p[2], *ap[2];
  float *xb;  // best iterate of the BiCGSTAB sweep (xr kernels keep it)
};

// p_new = r1 + beta (p_old - omega ap_old) (or r1 on restart, which also sets r0 = r1),
// evaluated at the stencil points; ap_new = A p_new; alpha = rho / <ap_new, r0>
__global__ void __launch_bounds__(kBlock) k32_pap(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                  SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float b = (float)sc->beta, w = (float)sc->omega;
  const bool rst = sc->restart != 0;
  const float *__restrict__ po = (parity ? v.p[1] : v.p[0]);
  const float *__restrict__ apo = (parity ? v.ap[1] : v.ap[0]);
  float *__restrict__ pn = (parity ? v.p[0] : v.p[1]);
  float *__restrict__ apn = (parity ? v.ap[0] : v.ap[1]);
  const float *__restrict__ r1 = v.r1;
  AccF acc;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    float pc;
    const float y = rst ? stencil_apply_diff(g, st, ic, jc, kc, row, [&](long long q) { return r1[q]; }, pc)
                        : stencil_apply_diff(g, st, ic, jc, kc, row,
                                               [&](long long q) { return r1[q] + b * (po[q] - w * apo[q]); }, pc);
    pn[row] = pc;
    apn[row] = y;
    float r0 = v.r0[row];
    if (rst) {
      r0 = r1[row];
      v.r0[row] = r0;
    }
    acc.add(y * r0);
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}

// s = r1 - alpha ap at the stencil points; as = A s; omega = <as, s> / <as, as>
__global__ void __launch_bounds__(kBlock) k32_sas(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                  SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float a = (float)sc->alpha;
  const float *__restrict__ ap = (parity ? v.ap[0] : v.ap[1]);
  const float *__restrict__ r1 = v.r1;
  AccF a0, a1;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    float sc_;
    const float y = stencil_apply_diff(g, st, ic, jc, kc, row, [&](long long q) { return r1[q] - a * ap[q]; }, sc_);
    v.s[row] = sc_;
    v.as[row] = y;
    a0.add(y * sc_);
    a1.add(y * y);
  }
  double acc[2] = {a0.get(), a1.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[2], out) && lin_tid() == 0) {
    double wv = out[0] / out[1];
    // s has vanished: the half step solved the system; omega = 0 makes the next kernel
    // take x += alpha p, r1 = s and stop instead of forming 0/0
    if (!(out[1] > 0.0 && isfinite(wv))) wv = 0.0;
    sc->omega = wv;
  }
}

// x += alpha p + omega s; r1 = s - omega as; stop test, beta, restart
__global__ void __launch_bounds__(kBlock) k32_xr(Geo g, Vec32 v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float a = (float)sc->alpha, w = (float)sc->omega;
  const float *__restrict__ p = (parity ? v.p[0] : v.p[1]);
  const bool keep = sc->snap != 0;  // the current x is the iterate to keep
  AccF n2, rr;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const float s = v.s[row];
    const float x = v.x[row];
    if (keep) v.xb[row] = x;
    v.x[row] = fmaf(w, s, fmaf(a, p[row], x));
    const float r1 = fmaf(-w, v.as[row], s);
    v.r1[row] = r1;
    n2.add(r1 * r1);
    rr.add(r1 * v.r0[row]);
  }
  double acc[2] = {n2.get(), rr.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[3], out)) {
    if (lin_tid() == 0) sc->par = parity ^ 1;  // this iteration's p and ap become the previous ones
    finish_iteration<true>(sc, out[0], out[1]);
  }
}

// ---- FP32 BiCGSTAB with a right preconditioner (the multigrid V-cycle, multigrid.cu) ----
// The iteration of bicgstabRe2 on A M y = r with x = M y: p and s are preconditioned
// (ph = M p, sh = M s) before each operator application and the update of x, while r, s,
// and the stop test stay on the unpreconditioned residual.  Same device scalars and
// decisions as the plain FP32 sweep (finish_iteration<true>), counters 1-3 as there.

// p = r1 + beta (p - omega v), or p = r0 = r1 on restart
__global__ void __launch_bounds__(kBlock) k32p_p(Geo g, PrecVecs v, const SolverScal *sc) {
  if (sc->done) return;
  const float b = (float)sc->beta, w = (float)sc->omega;
  const bool rst = sc->restart != 0;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const float r1 = v.r1[row];
    if (rst) {
      v.r0[row] = r1;
      v.p[row] = r1;
    } else {
      v.p[row] = r1 + b * (v.p[row] - w * v.v[row]);
    }
  }
}

// v = A ph, alpha = rho / <v, r0>
__global__ void __launch_bounds__(kBlock) k32p_v(Geo g, Stencil<float> st, PrecVecs v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const float *__restrict__ ph = v.ph;
  AccF acc;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    float c;
    const float y = stencil_apply_diff(g, st, ic, jc, kc, row, [&](long long q) { return ph[q]; }, c);
    v.v[row] = y;
    acc.add(y * v.r0[row]);
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}

// s = r1 - alpha v
__global__ void __launch_bounds__(kBlock) k32p_s(Geo g, PrecVecs v, const SolverScal *sc) {
  if (sc->done) return;
  const float a = (float)sc->alpha;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    v.s[row] = fmaf(-a, v.v[row], v.r1[row]);
  }
}

// t = A sh, omega = <t, s> / <t, t> (0 when t vanishes, as in k32_sas)
__global__ void __launch_bounds__(kBlock) k32p_t(Geo g, Stencil<float> st, PrecVecs v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const float *__restrict__ sh = v.sh;
  AccF a0, a1;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    float c;
    const float y = stencil_apply_diff(g, st, ic, jc, kc, row, [&](long long q) { return sh[q]; }, c);
    v.t[row] = y;
    a0.add(y * v.s[row]);
    a1.add(y * y);
  }
  double acc[2] = {a0.get(), a1.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[2], out) && lin_tid() == 0) {
    double wv = out[0] / out[1];
    if (!(out[1] > 0.0 && isfinite(wv))) wv = 0.0;
    sc->omega = wv;
  }
}

// x += alpha ph + omega sh; r1 = s - omega t; stop test, beta, restart
__global__ void __launch_bounds__(kBlock) k32p_xr(Geo g, PrecVecs v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const float a = (float)sc->alpha, w = (float)sc->omega;
  const bool keep = sc->snap != 0;
  AccF n2, rr;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const float x = v.x[row];
    if (keep) v.xb[row] = x;
    v.x[row] = fmaf(w, v.sh[row], fmaf(a, v.ph[row], x));
    const float r1 = fmaf(-w, v.t[row], v.s[row]);
    v.r1[row] = r1;
    n2.add(r1 * r1);
    rr.add(r1 * v.r0[row]);
  }
  double acc[2] = {n2.get(), rr.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[3], out)) finish_iteration<true>(sc, out[0], out[1]);
}

// ---- FP64 BiCGSTAB with the FP64 V-cycle as right preconditioner ----
// The FP32 preconditioned iteration above in FP64 (the like-for-like FP64 counterpart of
// the MIXED multigrid sweep): same kernels and order, FP64 vectors and dots.  Not the
// reference's iteration, so no rho-restart rule: it stops on the tolerance, the cap or a
// non-finite residual, and restarts only on a Lanczos breakdown.
__device__ __forceinline__ void finish_prec64(SolverScal *sc, double n2, double rr) {
  if (lin_tid() >= 32) return;
  const double tol = sc->tol, omega = sc->omega;
  const int iter = sc->iter + 1, maxit = sc->maxit;
  double relres, ao, rq;
  div3(sqrt(n2), sc->norm0, sc->alpha, omega, rr, sc->rho, relres, ao, rq);
  const double beta = ao * rq;
  if (lin_tid() != 0) return;
  sc->relres = relres;
  sc->iter = iter;
  if (!isfinite(relres)) {
    sc->done = 1;
    sc->status = CFDGB_ENAN;
  } else if (relres < tol) {
    sc->done = 1;
  } else if (iter >= maxit) {
    sc->done = 1;
    sc->status = CFDGB_ENOCONV;
  } else {
    sc->beta = beta;
    const bool broke = !(isfinite(beta) && omega != 0.0 && rr != 0.0);
    sc->restart = broke ? 1 : 0;
    sc->rho = broke ? n2 : rr;
  }
}

__global__ void __launch_bounds__(kBlock) k64p_p(Geo g, PrecVecsT<double> v, const SolverScal *sc) {
  if (sc->done) return;
  const double b = sc->beta, w = sc->omega;
  const bool rst = sc->restart != 0;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double r1 = v.r1[row];
    if (rst) {
      v.r0[row] = r1;
      v.p[row] = r1;
    } else {
      v.p[row] = fma(b, fma(-w, v.v[row], v.p[row]), r1);
    }
  }
}

__global__ void __launch_bounds__(kBlock) k64p_v(Geo g, Stencil<double> st, PrecVecsT<double> v, double *part,
                                                 SolverScal *sc) {
  if (sc->done) return;
  double a[1] = {0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double y = spmv_at<double>(g, st, v.ph, ic, jc, kc, row);
    v.v[row] = y;
    a[0] = fma(y, v.r0[row], a[0]);
  }
  double out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}

__global__ void __launch_bounds__(kBlock) k64p_s(Geo g, PrecVecsT<double> v, const SolverScal *sc) {
  if (sc->done) return;
  const double a = sc->alpha;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    v.s[row] = fma(-a, v.v[row], v.r1[row]);
  }
}

__global__ void __launch_bounds__(kBlock) k64p_t(Geo g, Stencil<double> st, PrecVecsT<double> v, double *part,
                                                 SolverScal *sc) {
  if (sc->done) return;
  double a[2] = {0.0, 0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double y = spmv_at<double>(g, st, v.sh, ic, jc, kc, row);
    v.t[row] = y;
    a[0] = fma(y, v.s[row], a[0]);
    a[1] = fma(y, y, a[1]);
  }
  double out[2];
  if (grid_sum<2>(a, part, &sc->cnt[2], out) && lin_tid() == 0) {
    double wv = out[0] / out[1];
    if (!(out[1] > 0.0 && isfinite(wv))) wv = 0.0;
    sc->omega = wv;
  }
}

__global__ void __launch_bounds__(kBlock) k64p_xr(Geo g, PrecVecsT<double> v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const double a = sc->alpha, w = sc->omega;
  double acc[2] = {0.0, 0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    v.x[row] = fma(w, v.sh[row], fma(a, v.ph[row], v.x[row]));
    const double r1 = fma(-w, v.t[row], v.s[row]);
    v.r1[row] = r1;
    acc[0] = fma(r1, r1, acc[0]);
    acc[1] = fma(r1, v.r0[row], acc[1]);
  }
  double out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[3], out)) finish_prec64(sc, out[0], out[1]);
}

// ---- FP32 iteration, vectorised: four consecutive k cells per thread (nzc % 4 == 0) ----
// One float4 load per vector and stencil point instead of four scalar loads; the k
// neighbours inside the quad come from registers.  Dot partials stay FP32 over the few
// dozen quads a thread owns and are added into the FP64 block/grid reduction once.
// k32v_xr is pointwise: a grid-stride loop over the planes.
#define FOR_QUADS(g)                                               \
  const int kc0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);     \
  const int kc = kc0; /* ROW(g) of the quad's first cell */        \
  const int jc = blockIdx.y * blockDim.y + threadIdx.y;            \
  const bool on_ = (kc0 < (g).nzc) && (jc < (g).nyc);              \
  for (int ic = blockIdx.z; on_ && ic < (g).nxc; ic += gridDim.z)

struct F4 {
  float v[4];
};
__device__ __forceinline__ F4 ld4(const float *p) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  return F4{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void st4(float *p, const F4 &a) {
  *reinterpret_cast<float4 *>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}

// The two stencil kernels march along x.  A thread owns one quad of one j row and walks a
// chunk of consecutive i planes (the same chunk for the whole block, so every thread runs
// the same trip count).  The values of planes i-1, i, i+1 stay in registers: per plane a
// thread loads the next plane's quad (its first read from HBM) and the quads of rows j-1
// and j+1 (L1 hits, loaded one plane earlier by their owners); the cells left and right
// of the quad come from the neighbouring lanes by warp shuffle, from memory only at a
// block's k edge.  f4(q) evaluates the stencil's argument at the quad of row q, f1(q) at
// one cell; body(row, centre values, A-applied values) consumes the result.  (A shared-
// memory tile for the j neighbours, one barrier per plane, measured slower.)
template <class F4f, class F1f, class Body>
__device__ __forceinline__ void march_quads(const Geo &g, const Stencil<float> &st, F4f &&f4, F1f &&f1, Body &&body) {
  const int kc0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  const int jc = blockIdx.y * blockDim.y + threadIdx.y;
  const bool on = kc0 < g.nzc && jc < g.nyc;
  const int chunk = (g.nxc + gridDim.z - 1) / gridDim.z;
  const int i0 = min(g.nxc, (int)blockIdx.z * chunk), i1 = min(g.nxc, i0 + chunk);
  const long long nyz = (long long)g.nyc * g.nzc;
  const bool hy0 = jc > 0, hy1 = jc + 1 < g.nyc;
  // cells left / right exist (periodic z: always, across the wrap at the line's ends)...
  const bool kl = kc0 > 0 || g.pz, kr = kc0 + 4 < g.nzc || g.pz;
  // ... and are held by the neighbouring lane (within the line)
  const bool sl = threadIdx.x > 0 && kc0 > 0, sr = threadIdx.x + 1 < blockDim.x && kc0 + 4 < g.nzc;
  const long long wl = kc0 > 0 ? -1 : g.nzc - 1, wr = kc0 + 4 < g.nzc ? 4 : 4 - g.nzc;  // their offsets
  long long row = ((long long)i0 * g.nyc + jc) * g.nzc + kc0;
  F4 fm{}, fc{};
  if (on && i0 < i1) {
    if (i0 > 0) fm = f4(row - nyz);
    fc = f4(row);
  }
  for (int ic = i0; ic < i1; ++ic, row += nyz) {
    F4 fp{}, ym{}, yp{};
    if (on) {
      if (ic + 1 < g.nxc) fp = f4(row + nyz);
      if (hy0) ym = f4(row - g.nzc);
      if (hy1) yp = f4(row + g.nzc);
    }
    const float l = __shfl_up_sync(0xffffffffu, fc.v[3], 1);
    const float r = __shfl_down_sync(0xffffffffu, fc.v[0], 1);
    const float zl = !kl ? 0.0f : (sl ? l : (on ? f1(row + wl) : 0.0f));
    const float zr = !kr ? 0.0f : (sr ? r : (on ? f1(row + wr) : 0.0f));
    // difference form (stencil_apply_diff); a missing neighbour has coefficient 0
    const int cxy = axis_class(ic, g.nxc) * 9 + axis_class(jc, g.nyc) * 3;
    const float *cmid = st.c[cxy + 1], *cfirst = st.c[cxy + (kc0 == 0 && !g.pz ? 0 : 1)],
                *clast = st.c[cxy + (kc0 + 4 == g.nzc && !g.pz ? 2 : 1)];
    F4 y;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float *c = q == 0 ? cfirst : (q == 3 ? clast : cmid);
      const float f0 = fc.v[q];
      const float zm = q == 0 ? zl : fc.v[q - 1], zp = q == 3 ? zr : fc.v[q + 1];
      float t = c[0] * (fm.v[q] - f0);
      t = fmaf(c[1], ym.v[q] - f0, t);
      t = fmaf(c[2], zm - f0, t);
      t = fmaf(c[4], zp - f0, t);
      t = fmaf(c[5], yp.v[q] - f0, t);
      t = fmaf(c[6], fp.v[q] - f0, t);
      y.v[q] = t;
    }
    if (on) body(row, fc, y);
    fm = fc;
    fc = fp;
  }
}

// march_quads for one vector f and an operand of the body, a plane further ahead: at plane i the
// loads of f at i + 2 and of the next plane's operand are issued, so that no plane waits for
// memory (28 -> 23 us on 512x256x64 for the preconditioned iteration's two operator kernels).
// Same quads a thread in the same order, same operations.
template <class Body>
__device__ __forceinline__ void march_quads_ahead(const Geo &g, const Stencil<float> &st, const float *__restrict__ f,
                                                  const float *__restrict__ opnd, Body &&body) {
  const int kc0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  const int jc = blockIdx.y * blockDim.y + threadIdx.y;
  const bool on = kc0 < g.nzc && jc < g.nyc;
  const int chunk = (g.nxc + gridDim.z - 1) / gridDim.z;
  const int i0 = min(g.nxc, (int)blockIdx.z * chunk), i1 = min(g.nxc, i0 + chunk);
  const long long nyz = (long long)g.nyc * g.nzc;
  const bool hy0 = jc > 0, hy1 = jc + 1 < g.nyc;
  const bool kl = kc0 > 0 || g.pz, kr = kc0 + 4 < g.nzc || g.pz;
  const bool sl = threadIdx.x > 0 && kc0 > 0, sr = threadIdx.x + 1 < blockDim.x && kc0 + 4 < g.nzc;
  const long long wl = kc0 > 0 ? -1 : g.nzc - 1, wr = kc0 + 4 < g.nzc ? 4 : 4 - g.nzc;
  const int cy = axis_class(jc, g.nyc) * 3, cz0 = kc0 == 0 && !g.pz ? 0 : 1, cz1 = kc0 + 4 == g.nzc && !g.pz ? 2 : 1;
  const float *q = f + (((long long)i0 * g.nyc + jc) * g.nzc + kc0);  // this plane's quad
  const float *o = opnd + (q - f);
  F4 fm{}, fc{}, fp{}, oc{};
  if (on && i0 < i1) {
    if (i0 > 0) fm = ld4(q - nyz);
    fc = ld4(q);
    if (i0 + 1 < g.nxc) fp = ld4(q + nyz);
    oc = ld4(o);
  }
  for (int ic = i0; ic < i1; ++ic, q += nyz, o += nyz) {
    F4 fn{}, on4{}, ym{}, yp{};
    if (on) {
      if (hy0) ym = ld4(q - g.nzc);
      if (hy1) yp = ld4(q + g.nzc);
      if (ic + 2 < g.nxc && ic + 1 < i1) fn = ld4(q + 2 * nyz);
      if (ic + 1 < i1) on4 = ld4(o + nyz);
    }
    const float l = __shfl_up_sync(0xffffffffu, fc.v[3], 1);
    const float r = __shfl_down_sync(0xffffffffu, fc.v[0], 1);
    const float zl = !kl ? 0.0f : (sl ? l : (on ? q[wl] : 0.0f));
    const float zr = !kr ? 0.0f : (sr ? r : (on ? q[wr] : 0.0f));
    const int cxy = axis_class(ic, g.nxc) * 9 + cy;
    const float *cmid = st.c[cxy + 1], *cfirst = st.c[cxy + cz0], *clast = st.c[cxy + cz1];
    F4 y;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float *c = t == 0 ? cfirst : (t == 3 ? clast : cmid);
      const float f0 = fc.v[t];
      const float zm = t == 0 ? zl : fc.v[t - 1], zp = t == 3 ? zr : fc.v[t + 1];
      float a = c[0] * (fm.v[t] - f0);
      a = fmaf(c[1], ym.v[t] - f0, a);
      a = fmaf(c[2], zm - f0, a);
      a = fmaf(c[4], zp - f0, a);
      a = fmaf(c[5], yp.v[t] - f0, a);
      a = fmaf(c[6], fp.v[t] - f0, a);
      y.v[t] = a;
    }
    if (on) body(q - f, y, oc);
    fm = fc;
    fc = fp;
    fp = fn;
    oc = on4;
  }
}

// p_new = r1 + beta (p_old - omega ap_old) (restart: p_new = r0 = r1); ap_new = A p_new;
// alpha = rho / <ap_new, r0>
__global__ void __launch_bounds__(kBlock) k32v_pap(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                   SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float b = (float)sc->beta, w = (float)sc->omega;
  const bool rst = sc->restart != 0;
  const float *__restrict__ po = (parity ? v.p[1] : v.p[0]);
  const float *__restrict__ apo = (parity ? v.ap[1] : v.ap[0]);
  float *__restrict__ pn = (parity ? v.p[0] : v.p[1]);
  float *__restrict__ apn = (parity ? v.ap[0] : v.ap[1]);
  const float *__restrict__ r1 = v.r1;
  float *__restrict__ r0 = v.r0;
  SumF acc;
  if (rst) {
    march_quads(
        g, st, [&](long long q) { return ld4(r1 + q); }, [&](long long q) { return r1[q]; },
        [&](long long row, const F4 &pc, const F4 &y) {
          st4(pn + row, pc);
          st4(apn + row, y);
          st4(r0 + row, pc);
#pragma unroll
          for (int t = 0; t < 4; ++t) acc.add(y.v[t], pc.v[t]);
        });
  } else {
    march_quads(
        g, st,
        [&](long long q) {
          const F4 r = ld4(r1 + q), p = ld4(po + q), a = ld4(apo + q);
          F4 o;
#pragma unroll
          for (int t = 0; t < 4; ++t) o.v[t] = fmaf(b, fmaf(-w, a.v[t], p.v[t]), r.v[t]);
          return o;
        },
        [&](long long q) { return fmaf(b, fmaf(-w, apo[q], po[q]), r1[q]); },
        [&](long long row, const F4 &pc, const F4 &y) {
          st4(pn + row, pc);
          st4(apn + row, y);
          const F4 z = ld4(r0 + row);
#pragma unroll
          for (int t = 0; t < 4; ++t) acc.add(y.v[t], z.v[t]);
        });
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}

// s = r1 - alpha ap; as = A s; omega = <as, s> / <as, as>
__global__ void __launch_bounds__(kBlock) k32v_sas(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                   SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float a = (float)sc->alpha;
  const float *__restrict__ ap = (parity ? v.ap[0] : v.ap[1]);
  const float *__restrict__ r1 = v.r1;
  float *__restrict__ sv = v.s;
  float *__restrict__ asv = v.as;
  SumF a0, a1;
  march_quads(
      g, st,
      [&](long long q) {
        const F4 r = ld4(r1 + q), p = ld4(ap + q);
        F4 o;
#pragma unroll
        for (int t = 0; t < 4; ++t) o.v[t] = fmaf(-a, p.v[t], r.v[t]);
        return o;
      },
      [&](long long q) { return fmaf(-a, ap[q], r1[q]); },
      [&](long long row, const F4 &s4, const F4 &y) {
        st4(sv + row, s4);
        st4(asv + row, y);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          a0.add(y.v[t], s4.v[t]);
          a1.add(y.v[t], y.v[t]);
        }
      });
  double acc[2] = {a0.get(), a1.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[2], out) && lin_tid() == 0) {
    double wv = out[0] / out[1];
    if (!(out[1] > 0.0 && isfinite(wv))) wv = 0.0;  // see k32_sas
    sc->omega = wv;
  }
}

// ---- the preconditioned FP32 iteration on quads (nzc % 4 == 0): the operator kernels march
// along x as k32v_sas does, the pointwise ones stride over float4 quads as k32v_xr does ----
__global__ void __launch_bounds__(kBlock) k32pv_p(Geo g, PrecVecs v, const SolverScal *sc) {
  if (sc->done) return;
  const float b = (float)sc->beta, w = (float)sc->omega;
  const bool rst = sc->restart != 0;
  const long long nq = g.ncell / 4, stride = (long long)gridDim.x * blockDim.x;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += stride) {
    const long long row = 4 * q;
    const F4 r1 = ld4(v.r1 + row);
    if (rst) {
      st4(v.r0 + row, r1);
      st4(v.p + row, r1);
      continue;
    }
    const F4 pp = ld4(v.p + row), vv = ld4(v.v + row);
    F4 o;
#pragma unroll
    for (int t = 0; t < 4; ++t) o.v[t] = r1.v[t] + b * (pp.v[t] - w * vv.v[t]);
    st4(v.p + row, o);
  }
}

__global__ void __launch_bounds__(kBlock) k32pv_v(Geo g, Stencil<float> st, PrecVecs v, double *part,
                                                  SolverScal *sc) {
  if (sc->done) return;
  const float *__restrict__ ph = v.ph;
  const float *__restrict__ r0 = v.r0;
  float *__restrict__ vv = v.v;
  SumF a0;
  march_quads_ahead(g, st, ph, r0, [&](long long row, const F4 &y, const F4 &r) {
    st4(vv + row, y);
#pragma unroll
    for (int t = 0; t < 4; ++t) a0.add(y.v[t], r.v[t]);
  });
  double a[1] = {a0.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}

__global__ void __launch_bounds__(kBlock) k32pv_s(Geo g, PrecVecs v, const SolverScal *sc) {
  if (sc->done) return;
  const float a = (float)sc->alpha;
  const long long nq = g.ncell / 4, stride = (long long)gridDim.x * blockDim.x;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += stride) {
    const long long row = 4 * q;
    const F4 r1 = ld4(v.r1 + row), vv = ld4(v.v + row);
    F4 o;
#pragma unroll
    for (int t = 0; t < 4; ++t) o.v[t] = fmaf(-a, vv.v[t], r1.v[t]);
    st4(v.s + row, o);
  }
}

__global__ void __launch_bounds__(kBlock) k32pv_t(Geo g, Stencil<float> st, PrecVecs v, double *part,
                                                  SolverScal *sc) {
  if (sc->done) return;
  const float *__restrict__ sh = v.sh;
  const float *__restrict__ sv = v.s;
  float *__restrict__ tv = v.t;
  SumF a0, a1;
  march_quads_ahead(g, st, sh, sv, [&](long long row, const F4 &y, const F4 &s4) {
    st4(tv + row, y);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      a0.add(y.v[t], s4.v[t]);
      a1.add(y.v[t], y.v[t]);
    }
  });
  double acc[2] = {a0.get(), a1.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[2], out) && lin_tid() == 0) {
    double wv = out[0] / out[1];
    if (!(out[1] > 0.0 && isfinite(wv))) wv = 0.0;
    sc->omega = wv;
  }
}

__global__ void __launch_bounds__(kBlock) k32pv_xr(Geo g, PrecVecs v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const float a = (float)sc->alpha, w = (float)sc->omega;
  const bool keep = sc->snap != 0;
  SumF n2, rr;
  const long long nq = g.ncell / 4, stride = (long long)gridDim.x * blockDim.x;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += stride) {
    const long long row = 4 * q;
    const F4 ph = ld4(v.ph + row), sh = ld4(v.sh + row), s = ld4(v.s + row), t4 = ld4(v.t + row),
             r0 = ld4(v.r0 + row);
    F4 x = ld4(v.x + row), r1;
    if (keep) st4(v.xb + row, x);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      x.v[t] = fmaf(w, sh.v[t], fmaf(a, ph.v[t], x.v[t]));
      r1.v[t] = fmaf(-w, t4.v[t], s.v[t]);
      n2.add(r1.v[t], r1.v[t]);
      rr.add(r1.v[t], r0.v[t]);
    }
    st4(v.x + row, x);
    st4(v.r1 + row, r1);
  }
  double acc[2] = {n2.get(), rr.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[3], out)) finish_iteration<true>(sc, out[0], out[1]);
}

// ---- FP32 stencil kernels on a bulk-copy (TMA) pipeline ----
// A block owns tj rows (all k) of the compact vectors and a chunk of consecutive i planes.
// Thread 0 streams each plane's rows jt-1 .. jt+tj (the halo rows included: one contiguous
// range per vector, since rows of a plane are contiguous) into one of kStages shared-memory
// stages with cp.async.bulk, signalling an mbarrier; every thread evaluates the stencil's
// argument from the stage, keeps its own quad's values of planes i-1, i, i+1 in registers
// and takes the j +- 1 values from the stage, the k +- 1 values by warp shuffle.  A stage is
// refilled once all warps have released it (a second mbarrier), one plane after its last
// use, so loads run up to kStages - 2 planes ahead of the computation.  Every wait is
// bounded: a wait that gives up sets sc->fault, the block stops, waits (bounded) for its
// own copies in flight and still joins the reduction.
constexpr int kStages = 4;
constexpr long long kWaitCycles = 1LL << 32;  // ~2 s at 2 GHz
constexpr long long kTestWaitCycles = 1LL << 20;  // ~0.5 ms: the wait limit of the test request

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// wait for the phase with the given parity to complete; false if it did not within `limit`
// cycles
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long limit = kWaitCycles) {
  const long long t0 = clock64();
  while (!mbar_test(bar, parity))
    if (clock64() - t0 > limit) return false;
  return true;
}
__device__ __forceinline__ void bulk_load(float *dst, const float *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// The vectors a stage holds: na with halo rows (the stencil's argument is built from them)
// and optionally one with the block's own rows only.
struct StageSrc {
  const float *a[3];
  int na;
  const float *own;
};

__host__ __device__ inline long long stage_floats(int tj, int nz, int na, bool own) {
  return (long long)na * (tj + 2) * nz + (own ? (long long)tj * nz : 0);
}

// fval(arrays of a stage, stage row, first cell) -> the argument's four values of a quad;
// f1(arrays, stage row, cell) -> one value; body(row, centre values, A-applied values,
// own-rows vector of the stage at this thread's row or nullptr)
template <class Fv, class F1, class Body>
__device__ __forceinline__ void tma_march(const Geo &g, const Stencil<float> &st, const StageSrc &src, SolverScal *sc,
                                          Fv &&fval, F1 &&f1, Body &&body) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int bad, test_wait;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);
  uint64_t *empty = full + kStages;
  float *stage0 = reinterpret_cast<float *>(smem + 128);
  const int nz = g.nzc, nq = nz / 4, tj = g.tj;
  const long long SA = (long long)(tj + 2) * nz, SS = stage_floats(tj, nz, src.na, src.own != nullptr);
  const int tid = threadIdx.x, lane = tid & 31;
  const int tq = tid % nq, ty = tid / nq;
  const int jt = blockIdx.x * tj, jc = jt + ty, kc0 = 4 * tq;
  const bool on = ty < tj && jc < g.nyc;
  const int chunk = (g.nxc + gridDim.y - 1) / gridDim.y;
  const int i0 = min(g.nxc, (int)blockIdx.y * chunk), i1 = min(g.nxc, i0 + chunk);
  if (i0 >= i1) return;  // uniform per block
  const int lo = max(i0 - 1, 0), hi = min(i1, g.nxc - 1), khi = hi - lo;  // staged planes lo..hi
  const int jlo = max(jt - 1, 0), jhi = min(jt + tj, g.nyc - 1), ohi = min(jt + tj, g.nyc) - 1;
  const uint32_t hbytes = (uint32_t)((jhi - jlo + 1) * nz * 4), obytes = (uint32_t)((ohi - jt + 1) * nz * 4);
  const uint32_t txb = src.na * hbytes + (src.own ? obytes : 0u);
  const long long nyz = (long long)g.nyc * nz;
  int issued = -1;  // thread 0: highest plane index issued
  auto issue = [&](int k) {
    const int s = k % kStages;
    float *dst = stage0 + s * SS;
    const long long plane = (long long)(lo + k) * nyz;
    // the test request announces 16 bytes more than plane 0's copies bring, so that wait
    // runs out (every copy issued still lands; nothing is left in flight)
    mbar_expect_tx(&full[s], txb + (k == 0 && test_wait ? 16u : 0u));
    for (int a = 0; a < src.na; ++a)
      bulk_load(dst + a * SA + (long long)(jlo - (jt - 1)) * nz, src.a[a] + plane + (long long)jlo * nz, hbytes,
                &full[s]);
    if (src.own) bulk_load(dst + src.na * SA, src.own + plane + (long long)jt * nz, obytes, &full[s]);
    issued = k;
  };
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kBlock / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    bad = 0;
    // a one-shot request (SolverScal::test_wait, set only by the host's test switch):
    // block (0,0) of the next pipelined launch takes it
    test_wait = 0;
    if (blockIdx.x == 0 && blockIdx.y == 0 && sc->test_wait) {
      sc->test_wait = 0;
      test_wait = 1;
    }
  }
  __syncthreads();
  const long long wait_limit = test_wait ? kTestWaitCycles : kWaitCycles;
  if (tid == 0)
    for (int k = 0; k <= min(khi, kStages - 1); ++k) issue(k);
  auto fail = [&]() {
    *(volatile int *)&bad = 1;
    atomicExch(&sc->fault, 1);
  };
  auto wait_full = [&](int k) {
    if (mbar_wait(&full[k % kStages], (k / kStages) & 1, wait_limit)) return true;
    fail();
    return false;
  };
  auto arrays = [&](int k) { return stage0 + (k % kStages) * SS; };
  auto release = [&](int k) {
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[k % kStages]);
  };
  auto refill = [&](int k) {  // thread 0: plane k was released by every warp -> load plane k + kStages
    if (tid != 0 || k < 0 || k + kStages > khi) return;
    if (!mbar_wait(&empty[k % kStages], (k / kStages) & 1, wait_limit)) {
      fail();
      return;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    issue(k + kStages);
  };
  const int own = ty + 1;  // this thread's stage row
  int kc = i0 - lo;        // stage index of the centre plane
  int waited = -1;         // highest plane this thread waited for
  bool ok = wait_full(0);
  waited = 0;
  F4 fm{}, fc{};
  if (ok && kc == 1) {
    ok = wait_full(1);
    waited = 1;
  }
  if (ok) {
    if (kc == 1) {
      if (on) fm = fval(arrays(0), own, kc0);
      release(0);
    }
    if (on) fc = fval(arrays(kc), own, kc0);
  }
  long long row = ((long long)i0 * g.nyc + jc) * nz + kc0;
  for (int ic = i0; ok && ic < i1; ++ic, ++kc, row += nyz) {
    if (*(volatile int *)&bad) {
      ok = false;
      break;
    }
    F4 fp{}, ym{}, yp{};
    if (ic + 1 < g.nxc) {
      if (!wait_full(kc + 1)) {
        ok = false;
        break;
      }
      waited = kc + 1;
      if (on) fp = fval(arrays(kc + 1), own, kc0);
    }
    const float *arr = arrays(kc);
    if (on) {
      if (jc > 0) ym = fval(arr, own - 1, kc0);
      if (jc + 1 < g.nyc) yp = fval(arr, own + 1, kc0);
    }
    const float l = __shfl_up_sync(0xffffffffu, fc.v[3], 1);
    const float r = __shfl_down_sync(0xffffffffu, fc.v[0], 1);
    // the cells left and right of the quad: from the neighbouring lane within the row, from
    // the stage at a warp's edge, across the wrap at the row's ends (periodic z), else none
    const float zl = (tq == 0 && !g.pz) ? 0.0f
                                       : ((lane > 0 && tq > 0) ? l : (on ? f1(arr, own, tq > 0 ? kc0 - 1 : nz - 1) : 0.0f));
    const float zr = (tq == nq - 1 && !g.pz)
                         ? 0.0f
                         : ((lane < 31 && tq < nq - 1) ? r : (on ? f1(arr, own, tq < nq - 1 ? kc0 + 4 : 0) : 0.0f));
    const int cxy = axis_class(ic, g.nxc) * 9 + axis_class(jc, g.nyc) * 3;
    const float *cmid = st.c[cxy + 1], *cfirst = st.c[cxy + (kc0 == 0 && !g.pz ? 0 : 1)],
                *clast = st.c[cxy + (kc0 + 4 == nz && !g.pz ? 2 : 1)];
    F4 y;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float *c = q == 0 ? cfirst : (q == 3 ? clast : cmid);
      const float f0 = fc.v[q];
      const float zm = q == 0 ? zl : fc.v[q - 1], zp = q == 3 ? zr : fc.v[q + 1];
      float t = c[0] * (fm.v[q] - f0);
      t = fmaf(c[1], ym.v[q] - f0, t);
      t = fmaf(c[2], zm - f0, t);
      t = fmaf(c[4], zp - f0, t);
      t = fmaf(c[5], yp.v[q] - f0, t);
      t = fmaf(c[6], fp.v[q] - f0, t);
      y.v[q] = t;
    }
    if (on) body(row, fc, y, src.own ? arr + src.na * SA + (long long)ty * nz + kc0 : nullptr);
    release(kc);
    refill(kc - 1);
    fm = fc;
    fc = fp;
  }
  if (!ok && tid == 0)  // stopped early: let this block's copies land before it exits
    for (int k = waited + 1; k <= issued; ++k) mbar_wait(&full[k % kStages], (k / kStages) & 1, wait_limit);
}

__device__ __forceinline__ F4 lds4(const float *p) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  return F4{{t.x, t.y, t.z, t.w}};
}

__global__ void __launch_bounds__(kBlock) k32t_pap(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                   SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float b = (float)sc->beta, w = (float)sc->omega;
  const bool rst = sc->restart != 0;
  const float *po = (parity ? v.p[1] : v.p[0]);
  const float *apo = (parity ? v.ap[1] : v.ap[0]);
  float *__restrict__ pn = (parity ? v.p[0] : v.p[1]);
  float *__restrict__ apn = (parity ? v.ap[0] : v.ap[1]);
  float *__restrict__ r0 = v.r0;
  const long long SA = (long long)(g.tj + 2) * g.nzc;
  const int nz = g.nzc;
  SumF acc;
  if (rst) {
    const StageSrc src{{v.r1, nullptr, nullptr}, 1, nullptr};
    tma_march(
        g, st, src, sc, [&](const float *a, int r, int k) { return lds4(a + r * nz + k); },
        [&](const float *a, int r, int k) { return a[r * nz + k]; },
        [&](long long row, const F4 &pc, const F4 &y, const float *) {
          st4(pn + row, pc);
          st4(apn + row, y);
          st4(r0 + row, pc);
#pragma unroll
          for (int t = 0; t < 4; ++t) acc.add(y.v[t], pc.v[t]);
        });
  } else {
    const StageSrc src{{v.r1, po, apo}, 3, r0};
    auto f4 = [&](const float *a, int r, int k) {
      const int o = r * nz + k;
      const F4 rr = lds4(a + o), pp = lds4(a + SA + o), aa = lds4(a + 2 * SA + o);
      F4 f;
#pragma unroll
      for (int t = 0; t < 4; ++t) f.v[t] = fmaf(b, fmaf(-w, aa.v[t], pp.v[t]), rr.v[t]);
      return f;
    };
    tma_march(
        g, st, src, sc, f4,
        [&](const float *a, int r, int k) {
          const int o = r * nz + k;
          return fmaf(b, fmaf(-w, a[2 * SA + o], a[SA + o]), a[o]);
        },
        [&](long long row, const F4 &pc, const F4 &y, const float *z0) {
          st4(pn + row, pc);
          st4(apn + row, y);
          const F4 z = lds4(z0);
#pragma unroll
          for (int t = 0; t < 4; ++t) acc.add(y.v[t], z.v[t]);
        });
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}

__global__ void __launch_bounds__(kBlock) k32t_sas(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                   SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float al = (float)sc->alpha;
  const float *ap = (parity ? v.ap[0] : v.ap[1]);
  float *__restrict__ sv = v.s;
  float *__restrict__ asv = v.as;
  const long long SA = (long long)(g.tj + 2) * g.nzc;
  const int nz = g.nzc;
  SumF a0, a1;
  const StageSrc src{{v.r1, ap, nullptr}, 2, nullptr};
  tma_march(
      g, st, src, sc,
      [&](const float *a, int r, int k) {
        const int o = r * nz + k;
        const F4 rr = lds4(a + o), pp = lds4(a + SA + o);
        F4 f;
#pragma unroll
        for (int t = 0; t < 4; ++t) f.v[t] = fmaf(-al, pp.v[t], rr.v[t]);
        return f;
      },
      [&](const float *a, int r, int k) { return fmaf(-al, a[SA + r * nz + k], a[r * nz + k]); },
      [&](long long row, const F4 &s4, const F4 &y, const float *) {
        st4(sv + row, s4);
        st4(asv + row, y);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          a0.add(y.v[t], s4.v[t]);
          a1.add(y.v[t], y.v[t]);
        }
      });
  double acc[2] = {a0.get(), a1.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[2], out) && lin_tid() == 0) {
    double wv = out[0] / out[1];
    if (!(out[1] > 0.0 && isfinite(wv))) wv = 0.0;  // see k32_sas
    sc->omega = wv;
  }
}

// Shared memory of the bulk-copy kernels and their residency.  The pap kernel stages three
// vectors with halo rows and one without; the two-vector kernels (sas, CG pq) stage two, so
// they get their own, smaller size and more resident blocks.  0 when the grid does not fit
// the scheme (nz % 4 != 0 or more than 256 quads per row).
__global__ void k32cgt_pq(Geo g, Stencil<float> st, Vec32 v, double *part, SolverScal *sc);

int fp32_stage_plan(int nzc, int *tj, int *smem_bytes, int *blocks_per_sm, int *smem2_bytes, int *blocks2_per_sm) {
  if (nzc % 4 != 0 || nzc / 4 > kBlock) return 0;
  const int t = kBlock / (nzc / 4);
  const long long bytes = 128 + kStages * stage_floats(t, nzc, 3, true) * 4;
  const long long bytes2 = 128 + kStages * stage_floats(t, nzc, 2, false) * 4;
  if (bytes > 227 * 1024) return 0;
  *tj = t;
  *smem_bytes = (int)bytes;
  *smem2_bytes = (int)bytes2;
  if (cudaFuncSetAttribute(k32t_pap, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess ||
      cudaFuncSetAttribute(k32t_sas, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes2) != cudaSuccess ||
      cudaFuncSetAttribute(k32cgt_pq, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes2) != cudaSuccess)
    return 0;
  int n = 0, n2 = 0, n3 = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k32t_pap, kBlock, (size_t)bytes) != cudaSuccess || n < 1 ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n2, k32t_sas, kBlock, (size_t)bytes2) != cudaSuccess || n2 < 1 ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n3, k32cgt_pq, kBlock, (size_t)bytes2) != cudaSuccess || n3 < 1)
    return 0;
  *blocks_per_sm = n;
  *blocks2_per_sm = n2 < n3 ? n2 : n3;
  return 1;
}

// x += alpha p + omega s; r1 = s - omega as; ||r1||^2, <r1, r0>.  Pointwise, so a flat
// grid-stride loop over quads with a grid sized to fill every SM (g.xgrid blocks).
__global__ void __launch_bounds__(kBlock) k32v_xr(Geo g, Vec32 v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float a = (float)sc->alpha, w = (float)sc->omega;
  const float *__restrict__ p = (parity ? v.p[0] : v.p[1]);
  const float *__restrict__ sv = v.s;
  const float *__restrict__ asv = v.as;
  const float *__restrict__ r0v = v.r0;
  float *__restrict__ xv = v.x;
  float *__restrict__ r1v = v.r1;
  float *__restrict__ xb = v.xb;
  const bool keep = sc->snap != 0;  // the current x is the iterate to keep
  SumF n2, rr;
  const long long nq = g.ncell / 4, stride = (long long)gridDim.x * blockDim.x;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += stride) {
    const long long row = 4 * q;
    const F4 s = ld4(sv + row), as = ld4(asv + row), pp = ld4(p + row), r0 = ld4(r0v + row);
    F4 x = ld4(xv + row), r1;
    if (keep) st4(xb + row, x);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      x.v[t] = fmaf(w, s.v[t], fmaf(a, pp.v[t], x.v[t]));
      r1.v[t] = fmaf(-w, as.v[t], s.v[t]);
      n2.add(r1.v[t], r1.v[t]);
      rr.add(r1.v[t], r0.v[t]);
    }
    st4(xv + row, x);
    st4(r1v + row, r1);
  }
  double acc[2] = {n2.get(), rr.get()}, out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[3], out)) {
    if (lin_tid() == 0) sc->par = parity ^ 1;  // this iteration's p and ap become the previous ones
    finish_iteration<true>(sc, out[0], out[1]);
  }
}

__global__ void k32cg_xr(Geo g, Vec32 v, double *part, SolverScal *sc);

int fp32_pointwise_blocks_per_sm() {
  // the grid serves both pointwise kernels (BiCGSTAB and CG sweeps): the smaller residency
  int a = 0, b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k32v_xr, kBlock, 0) != cudaSuccess) a = 4;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k32cg_xr, kBlock, 0) != cudaSuccess) b = 4;
  const int n = a < b ? a : b;
  return n > 0 ? n : 1;
}

// ---- conjugate gradients on the SPE operator ----
// The reference's other Krylov solver, inc/solver/cg.hpp (selected by P_SOLVER_CG_ELL):
// unpreconditioned CG, x += alpha p, r -= alpha q, beta = <r, r>_new / <r, r>_old.  (That
// header does not compile as published; the method it spells out is followed, with
// bicgstabRe2's stop test ||r|| / ||b|| < tol and iteration cap.)  Three FP64 kernels per
// iteration; the FP32 sweeps of the MIXED mode fuse the p update into the SpMV (two
// kernels, 10 words per cell).
__device__ __forceinline__ void finish_cg64(SolverScal *sc, double n2) {
  if (lin_tid() >= 32) return;
  const double tol = sc->tol;
  const int iter = sc->iter, maxit = sc->maxit;
  double relres, beta, unused;
  div3(sqrt(n2), sc->norm0, n2, sc->rho, n2, sc->rho, relres, beta, unused);
  if (lin_tid() != 0) return;
  sc->relres = relres;
  if (relres < tol) {
    sc->done = 1;
  } else if (!isfinite(relres)) {
    sc->done = 1;
    sc->status = CFDGB_ENAN;
  } else if (iter >= maxit) {
    sc->done = 1;
    sc->status = CFDGB_ENOCONV;
  } else {
    sc->beta = beta;
    sc->rho = n2;
    sc->iter = iter + 1;
  }
}

// r = b - A x, p = r; history px2 <- px1 <- x (the NaN recovery of the BiCGSTAB path)
__global__ void __launch_bounds__(kBlock) k64cg_setup(Geo g, Stencil<double> st, KrylovVecs<double> v,
                                                       const double *__restrict__ b, double *px1, double *px2,
                                                       double *part, SolverScal *sc) {
  double acc[2] = {0.0, 0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double bb = b[row];
    const double r = bb - spmv_at<double>(g, st, v.x, ic, jc, kc, row);
    v.r1[row] = r;
    v.p1[row] = r;
    px2[row] = px1[row];
    px1[row] = v.x[row];
    acc[0] += bb * bb;
    acc[1] += r * r;
  }
  double out[2];
  if (grid_sum<2>(acc, part, &sc->cnt[0], out) && lin_tid() == 0) {
    sc->timestep += 1;
    sc->norm0 = sqrt(out[0]);
    sc->rho = out[1];
    sc->iter = 0;
    sc->status = 0;
    sc->fault = 0;
    sc->relres = sqrt(out[1]) / sc->norm0;
    sc->done = (sc->relres < sc->tol) ? 1 : 0;
  }
}
// q = A p, alpha = rho / <p, q>
__global__ void __launch_bounds__(kBlock) k64cg_q(Geo g, Stencil<double> st, KrylovVecs<double> v, double *part,
                                                   SolverScal *sc) {
  if (sc->done) return;
  double a[1] = {0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double q = spmv_at<double>(g, st, v.p1, ic, jc, kc, row);
    v.ap[row] = q;
    a[0] += q * v.p1[row];
  }
  double out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}
// x += alpha p, r -= alpha q, ||r||^2: stop test and beta
__global__ void __launch_bounds__(kBlock) k64cg_xr(Geo g, KrylovVecs<double> v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const double al = sc->alpha;
  double a[1] = {0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    v.x[row] = fma(al, v.p1[row], v.x[row]);
    const double r = fma(-al, v.ap[row], v.r1[row]);
    v.r1[row] = r;
    a[0] += r * r;
  }
  double out[1];
  if (grid_sum<1>(a, part, &sc->cnt[3], out)) finish_cg64(sc, out[0]);
}
// p = r + beta p
__global__ void __launch_bounds__(kBlock) k64cg_p(Geo g, KrylovVecs<double> v, const SolverScal *sc) {
  if (sc->done) return;
  const double be = sc->beta;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    v.p1[row] = fma(be, v.p1[row], v.r1[row]);
  }
}

// FP32 sweep (MIXED): hand over to the FP64 refinement like the BiCGSTAB sweeps
__device__ __forceinline__ void finish_cg32(SolverScal *sc, double n2) {
  if (lin_tid() >= 32) return;
  const double tol = sc->tol, best = sc->best, delta = sc->delta, rmax = sc->rmax, rn = sqrt(n2);
  const int iter = sc->iter, maxit = sc->maxit;
  double relres, beta, unused;
  div3(rn, sc->norm0, n2, sc->rho, n2, sc->rho, relres, beta, unused);
  if (lin_tid() != 0) return;
  sc->relres = relres;
  if (relres < best) sc->best = relres;
  if (!isfinite(relres)) {
    sc->done = 1;
    sc->status = CFDGB_ENAN;
  } else if (iter > 16 && relres > 1e3 * (relres < best ? relres : best)) {
    sc->done = 1;
    sc->status = CFDGB_ENOCONV;
  } else if (iter >= maxit) {
    sc->done = 1;
    sc->status = CFDGB_ENOCONV;
    sc->iter = iter + 1;
  } else if (relres < tol || rn < delta * rmax) {
    sc->done = 1;
    sc->status = kStatusRefine;
    sc->iter = iter + 1;
  } else {
    sc->beta = beta;
    sc->rho = n2;
    sc->restart = isfinite(beta) ? 0 : 1;
    sc->rmax = fmax(rmax, rn);
    sc->iter = iter + 1;
  }
}

// p_new = r + beta p_old (restart: r) at the stencil points; q = A p_new; alpha = rho / <p_new, q>
__global__ void __launch_bounds__(kBlock) k32cgt_pq(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                     SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float be = (float)sc->beta;
  const bool rst = sc->restart != 0;
  const float *po = (parity ? v.p[1] : v.p[0]);
  float *__restrict__ pn = (parity ? v.p[0] : v.p[1]);
  float *__restrict__ q = v.ap[0];
  const long long SA = (long long)(g.tj + 2) * g.nzc;
  const int nz = g.nzc;
  SumF acc;
  auto body = [&](long long row, const F4 &pc, const F4 &y, const float *) {
    st4(pn + row, pc);
    st4(q + row, y);
#pragma unroll
    for (int t = 0; t < 4; ++t) acc.add(y.v[t], pc.v[t]);
  };
  if (rst) {
    const StageSrc src{{v.r1, nullptr, nullptr}, 1, nullptr};
    tma_march(
        g, st, src, sc, [&](const float *a, int r, int k) { return lds4(a + r * nz + k); },
        [&](const float *a, int r, int k) { return a[r * nz + k]; }, body);
  } else {
    const StageSrc src{{v.r1, po, nullptr}, 2, nullptr};
    tma_march(
        g, st, src, sc,
        [&](const float *a, int r, int k) {
          const int o = r * nz + k;
          const F4 rr = lds4(a + o), pp = lds4(a + SA + o);
          F4 f;
#pragma unroll
          for (int t = 0; t < 4; ++t) f.v[t] = fmaf(be, pp.v[t], rr.v[t]);
          return f;
        },
        [&](const float *a, int r, int k) { return fmaf(be, a[SA + r * nz + k], a[r * nz + k]); }, body);
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}
__global__ void __launch_bounds__(kBlock) k32cgv_pq(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                     SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float be = (float)sc->beta;
  const bool rst = sc->restart != 0;
  const float *__restrict__ po = (parity ? v.p[1] : v.p[0]);
  float *__restrict__ pn = (parity ? v.p[0] : v.p[1]);
  float *__restrict__ q = v.ap[0];
  const float *__restrict__ r1 = v.r1;
  SumF acc;
  auto body = [&](long long row, const F4 &pc, const F4 &y) {
    st4(pn + row, pc);
    st4(q + row, y);
#pragma unroll
    for (int t = 0; t < 4; ++t) acc.add(y.v[t], pc.v[t]);
  };
  if (rst) {
    march_quads(
        g, st, [&](long long k) { return ld4(r1 + k); }, [&](long long k) { return r1[k]; }, body);
  } else {
    march_quads(
        g, st,
        [&](long long k) {
          const F4 rr = ld4(r1 + k), pp = ld4(po + k);
          F4 f;
#pragma unroll
          for (int t = 0; t < 4; ++t) f.v[t] = fmaf(be, pp.v[t], rr.v[t]);
          return f;
        },
        [&](long long k) { return fmaf(be, po[k], r1[k]); }, body);
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}
__global__ void __launch_bounds__(kBlock) k32cg_pq(Geo g, Stencil<float> st, Vec32 v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float be = (float)sc->beta;
  const bool rst = sc->restart != 0;
  const float *__restrict__ po = (parity ? v.p[1] : v.p[0]);
  float *__restrict__ pn = (parity ? v.p[0] : v.p[1]);
  const float *__restrict__ r1 = v.r1;
  AccF acc;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    float pc;
    const float y = rst ? stencil_apply_diff(g, st, ic, jc, kc, row, [&](long long k) { return r1[k]; }, pc)
                        : stencil_apply_diff(g, st, ic, jc, kc, row,
                                             [&](long long k) { return fmaf(be, po[k], r1[k]); }, pc);
    pn[row] = pc;
    v.ap[0][row] = y;
    acc.add(y * pc);
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[1], out) && lin_tid() == 0) sc->alpha = sc->rho / out[0];
}
// x += alpha p_new; r -= alpha q; ||r||^2: refinement test and beta (flat: any cell count)
__global__ void __launch_bounds__(kBlock) k32cg_xr(Geo g, Vec32 v, double *part, SolverScal *sc) {
  if (sc->done) return;
  const int parity = sc->par;
  const float al = (float)sc->alpha;
  const float *__restrict__ p = (parity ? v.p[0] : v.p[1]);
  const float *__restrict__ q = v.ap[0];
  float *__restrict__ xv = v.x;
  float *__restrict__ r1v = v.r1;
  SumF n2;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g.ncell % 4 == 0) {
    for (long long k = t0; k < g.ncell / 4; k += stride) {
      const long long row = 4 * k;
      const F4 pp = ld4(p + row), qq = ld4(q + row);
      F4 x = ld4(xv + row), r = ld4(r1v + row);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        x.v[t] = fmaf(al, pp.v[t], x.v[t]);
        r.v[t] = fmaf(-al, qq.v[t], r.v[t]);
        n2.add(r.v[t], r.v[t]);
      }
      st4(xv + row, x);
      st4(r1v + row, r);
    }
  } else {
    for (long long row = t0; row < g.ncell; row += stride) {
      xv[row] = fmaf(al, p[row], xv[row]);
      const float r = fmaf(-al, q[row], r1v[row]);
      r1v[row] = r;
      n2.add(r, r);
    }
  }
  double acc[1] = {n2.get()}, out[1];
  if (grid_sum<1>(acc, part, &sc->cnt[3], out)) {
    if (lin_tid() == 0) sc->par = parity ^ 1;
    finish_cg32(sc, out[0]);
  }
}

// ---- FP64 Krylov iterations in one cooperative launch ----
// On grids up to a few million cells an iteration's kernels are short (2-20 us) and mostly
// latency: each launch ramps up, reads its scalars through L2 and three of five end in a
// reduction whose last block works alone.  Here one block a multiprocessor keeps a contiguous
// range of cells for the whole chunk of iterations; the phases of an iteration (the five
// kernels above, or CG's three) are separated by a grid barrier of one counter, and after a
// reducing phase every block sums the block partials itself, in the same order, so the
// scalars need no second round trip.  Same operations per cell as the kernels above; the dot
// products are summed in this partition's order.
// Measured, us an iteration, a kernel a phase -> one launch: BiCGSTAB 18 K cells 26 -> 11.7, 1.05 M
// 76 -> 61 (the FP64 pipe's time is 41.7), stretched 1.6 M 118 -> 83; CG 314 K 24.7 -> 15.6.
// The barrier counts arrivals (sc->cnt[6], back to zero through sc->cnt[7] when the last block
// leaves).  A wait is bounded: a block whose wait gives up leaves with a mark in the second counter,
// and so do the others, each after its own bounded wait; the last one out turns it into sc->fault and
// CFDGB_ECUDA.  (Polling all blocks' sums, each word tagged with the reduction's number, instead of the
// counter: 152 x 152 polled words slow the stores they wait for, 96x48x4 12.7 -> 23.7 us an iteration:
// not kept.)
constexpr int kLoopBlock = 512;
constexpr int kLoopMaxBlocks = 512;  // the most blocks whose sums a slot holds
constexpr long long kLoopWaitCycles = 1LL << 32;  // ~2 s
constexpr int kLoopSlots = 5;        // values reduced in an iteration

struct LoopScal {
  double rho, alpha, omega, beta, relres, best, rmax;
  int iter, done, status, restart, bad;
};

struct LoopGrid {
  SolverScal *sc;
  double *part;     // [slot][kLoopMaxBlocks]
  unsigned target;  // arrivals that complete the next barrier
  long long limit;  // cycles a wait may take
  // one thread: this block's arrival, and the wait for all (the block's stores come before, by the
  // barrier that its threads passed)
  __device__ __forceinline__ void arrive_wait(LoopScal &L) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&sc->cnt[6]) : "memory");
    const long long t0 = clock64();
    for (;;) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&sc->cnt[6]) : "memory");
      if ((int)(v - target) >= 0) break;
      if (clock64() - t0 > limit) {
        L.bad = 1;
        break;
      }
    }
  }
  __device__ __forceinline__ bool sync(LoopScal &L) {
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) arrive_wait(L);
    __syncthreads();
    return L.bad == 0;
  }
  // sums of v over the grid (slots s..), with a barrier; warp 0 calls fin(sums) in all its lanes,
  // which leaves the scalars in L.  Warp 0 alone adds up its block, arrives, waits and adds up the
  // blocks, each of its lanes a few of them: two block barriers in all
  template <int NV, class Fin>
  __device__ __forceinline__ bool reduce(LoopScal &L, double (&v)[NV], int s, Fin &&fin) {
    __shared__ double sh[NV][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
    warp_sum<NV>(v);
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < NV; ++q) sh[q][wid] = v[q];
    target += gridDim.x;
    __syncthreads();
    if (wid == 0) {
      double o[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) o[q] = warp_sum1(lane < nw ? sh[q][lane] : 0.0);
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) part[(s + q) * kLoopMaxBlocks + blockIdx.x] = o[q];
        arrive_wait(L);
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < NV; ++q) o[q] = 0.0;
      for (int b0 = 0; b0 < (int)gridDim.x; b0 += 160) {
        double t[NV][5];
#pragma unroll
        for (int q = 0; q < NV; ++q)
#pragma unroll
          for (int e = 0; e < 5; ++e) {
            const int b = b0 + 32 * e + lane;
            t[q][e] = b < (int)gridDim.x ? __ldcg(part + (s + q) * kLoopMaxBlocks + b) : 0.0;
          }
#pragma unroll
        for (int q = 0; q < NV; ++q) o[q] += (t[q][0] + (t[q][1] + t[q][2])) + (t[q][3] + t[q][4]);
      }
#pragma unroll
      for (int q = 0; q < NV; ++q) o[q] = warp_sum1(o[q]);
      if (L.bad == 0) fin(o);
    }
    __syncthreads();
    return L.bad == 0;
  }
};

// The test request (sc->test_wait, set only by the host's test switch): block 0 waits for one
// arrival too many, every block with a short limit, so that its wait at the chunk's last barrier runs
// out
__device__ __forceinline__ LoopGrid loop_grid(SolverScal *sc, double *part) {
  const int test = sc->test_wait;
  return LoopGrid{sc, part, test && blockIdx.x == 0 ? 1u : 0u, test ? kTestWaitCycles : kLoopWaitCycles};
}
// scalars in, and out by block 0 when every block has left the loop's last barrier
__device__ __forceinline__ void loop_begin(LoopScal &L, const SolverScal *sc) {
  if (threadIdx.x == 0) {
    L.rho = sc->rho;
    L.alpha = sc->alpha;
    L.omega = sc->omega;
    L.beta = sc->beta;
    L.relres = sc->relres;
    L.best = sc->best;
    L.rmax = sc->rmax;
    L.iter = sc->iter;
    L.done = sc->done;
    L.status = sc->status;
    L.restart = sc->restart;
    L.bad = 0;
  }
  __syncthreads();
}
__device__ __forceinline__ void loop_end(const LoopScal &L, const LoopGrid &G) {
  SolverScal *const sc = G.sc;
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (L.bad == 0 && blockIdx.x == 0) {
    sc->rho = L.rho;
    sc->alpha = L.alpha;
    sc->omega = L.omega;
    sc->beta = L.beta;
    sc->relres = L.relres;
    sc->best = L.best;
    sc->rmax = L.rmax;
    sc->iter = L.iter;
    sc->done = L.done;
    sc->status = L.status;
    sc->restart = L.restart;
  }
  __threadfence();
  // blocks that left, and above them those whose wait gave up
  const unsigned own = L.bad ? kLoopGaveUp + 1u : 1u, left = atomicAdd(&sc->cnt[7], own) + own;
  if ((left & (kLoopGaveUp - 1u)) == gridDim.x) {  // every block is past its last wait
    if (left >= kLoopGaveUp) {  // over what block 0 left: its own waits may all have ended
      __threadfence();
      sc->fault = 1;
      sc->status = CFDGB_ECUDA;
      sc->done = 1;
      sc->test_wait = 0;
    }
    sc->cnt[6] = 0u;
    sc->cnt[7] = 0u;
  }
}

// finish_iteration<false> on the loop's scalars (warp 0)
__device__ __forceinline__ void loop_finish(LoopScal &L, double norm0, double tol, double thr, int maxit, int timestep,
                                            double n2, double rr) {
  const double rho_old = L.rho;
  double relres, ao, rq;
  div3(sqrt(n2), norm0, L.alpha, L.omega, rr, rho_old, relres, ao, rq);
  if (threadIdx.x != 0) return;
  L.relres = relres;
  if (relres < tol) {
    L.done = 1;
  } else if (L.iter >= maxit) {
    L.done = 1;
    L.status = CFDGB_ENOCONV;
  } else {
    L.rho = rr;
    L.beta = ao * rq;
    L.restart = !(timestep < 10 || fabs(rho_old) > thr);
    L.iter += 1;
  }
}

// The cells of a block: a contiguous range, the threads strided through it.  load(row) reads a
// cell's values and use(row, values) consumes them; the next cell's loads are issued before
// this one's arithmetic (a block a multiprocessor has too few warps to hide L2's latency with).
template <class Load, class Use>
__device__ __forceinline__ void loop_cells(long long lo, long long hi, Load &&load, Use &&use) {
  long long row = lo + threadIdx.x;
  if (row >= hi) return;
  auto cur = load(row);
  for (;;) {
    const long long next = row + kLoopBlock;
    if (next >= hi) break;
    auto nxt = load(next);
    use(row, cur);
    cur = nxt;
    row = next;
  }
  use(row, cur);
}
template <int N>
struct LoopVals {
  double v[N];
};

// The operator at a row: the neighbours' values in the order of stencil_apply's terms (zero
// where there is none), the centre, and what the row's entries need.  MODE 0: a uniform grid
// (class table).  The stretched grid takes its entries from the per-axis factors and one stored
// value a row (jp, or SPE's diagonal) instead of the seven stored entries, which were 56 bytes
// a cell and application: MODE 1, Jacobi-scaled rows, f_c - jp sum(factor f_nb) (the diagonal
// dj jp is 1 to within half an ulp, as jp = RN(1/dj)); MODE 2, SPE rows.
struct LoopStencil {
  double f[6], c, d, z;
  int ic, jc, kc;
};
template <int MODE>
__device__ __forceinline__ LoopStencil loop_load(const Geo &g, const double *f, const double *z, long long row) {
  LoopStencil S;
  row_cijk(row, g.nyc, g.nzc, S.ic, S.jc, S.kc);
  const long long nyz = (long long)g.nyc * g.nzc, zm = z_minus(g, S.kc, row), zp = z_plus(g, S.kc, row);
  S.f[0] = S.ic > 0 ? f[row - nyz] : 0.0;
  S.f[1] = S.jc > 0 ? f[row - g.nzc] : 0.0;
  S.f[2] = zm >= 0 ? f[zm] : 0.0;
  S.f[3] = zp >= 0 ? f[zp] : 0.0;
  S.f[4] = S.jc < g.nyc - 1 ? f[row + g.nzc] : 0.0;
  S.f[5] = S.ic < g.nxc - 1 ? f[row + nyz] : 0.0;
  S.c = f[row];
  if (z) S.z = z[row];
  if (MODE == 1) S.d = g.jpv[row];
  if (MODE == 2) S.d = g.cof[0][3 * g.ncell + row];
  return S;
}
template <int MODE>
__device__ __forceinline__ double loop_apply(const Geo &g, const Stencil<double> &st, const LoopStencil &S) {
  if (MODE == 0) {
    const double *c = st.c[cls_of(g, S.ic, S.jc, S.kc)];
    double y = c[0] * S.f[0];
    y = fma(c[1], S.f[1], y);
    y = fma(c[2], S.f[2], y);
    y = fma(c[3], S.c, y);
    y = fma(c[4], S.f[3], y);
    y = fma(c[5], S.f[4], y);
    return fma(c[6], S.f[5], y);
  }
  const double *ym = MODE == 1 ? g.fym : g.fyp, *yp = MODE == 1 ? g.fyp : g.fym;  // SPE_sparseMatrix.hpp:79,83
  double y = g.fxm[S.ic] * S.f[0];
  y = fma(ym[S.jc], S.f[1], y);
  y = fma(g.fzm[S.kc], S.f[2], y);
  y = fma(g.fzp[S.kc], S.f[3], y);
  y = fma(yp[S.jc], S.f[4], y);
  y = fma(g.fxp[S.ic], S.f[5], y);
  return MODE == 1 ? fma(-S.d, y, S.c) : fma(S.d, S.c, -y);
}

template <int MODE>
__global__ void __launch_bounds__(kLoopBlock, 1) k64_bicg_loop(Geo g, Stencil<double> st, KrylovVecs<double> v,
                                                               double *part, SolverScal *sc, int iters, int chunk) {
  __shared__ LoopScal L;
  loop_begin(L, sc);
  if (L.done) return;  // the same in every block: sc is written only after the last barrier
  LoopGrid G = loop_grid(sc, part);
  const double norm0 = sc->norm0, tol = sc->tol, thr = sc->restart_thr;
  const int maxit = sc->maxit, timestep = sc->timestep;
  const long long lo = min(g.ncell, (long long)blockIdx.x * chunk), hi = min(g.ncell, lo + chunk);
  double *x = v.x, *r0 = v.r0, *r1 = v.r1, *p1 = v.p1, *s = v.s, *ap = v.ap, *as = v.as;
  for (int it = 0; it < iters; ++it) {
    {  // ap = A p1, alpha
      double a[1] = {0.0};
      loop_cells(
          lo, hi, [&](long long row) { return loop_load<MODE>(g, p1, r0, row); },
          [&](long long row, const LoopStencil &S) {
            const double y = loop_apply<MODE>(g, st, S);
            ap[row] = y;
            a[0] = fma(y, S.z, a[0]);
          });
      if (!G.reduce<1>(L, a, 0, [&](const double (&o)[1]) {
            const double al = L.rho / o[0];
            if (threadIdx.x == 0) L.alpha = al;
          }))
        break;
    }
    const double al = L.alpha;
    loop_cells(
        lo, hi, [&](long long row) { return LoopVals<2>{{r1[row], ap[row]}}; },
        [&](long long row, const LoopVals<2> &q) { s[row] = fma(-al, q.v[1], q.v[0]); });
    if (!G.sync(L)) break;
    {  // as = A s, omega
      double a[2] = {0.0, 0.0};
      loop_cells(
          lo, hi, [&](long long row) { return loop_load<MODE>(g, s, nullptr, row); },
          [&](long long row, const LoopStencil &S) {
            const double y = loop_apply<MODE>(g, st, S);
            as[row] = y;
            a[0] = fma(y, S.c, a[0]);
            a[1] = fma(y, y, a[1]);
          });
      if (!G.reduce<2>(L, a, 1, [&](const double (&o)[2]) {
            const double w = o[0] / o[1];
            if (threadIdx.x == 0) L.omega = w;
          }))
        break;
    }
    const double w = L.omega;
    {  // x, r1, stop test and beta
      double a[2] = {0.0, 0.0};
      loop_cells(
          lo, hi, [&](long long row) { return LoopVals<5>{{s[row], as[row], p1[row], x[row], r0[row]}}; },
          [&](long long row, const LoopVals<5> &q) {
            const double r = fma(-w, q.v[1], q.v[0]);
            x[row] = fma(w, q.v[0], fma(al, q.v[2], q.v[3]));
            r1[row] = r;
            a[0] = fma(r, r, a[0]);
            a[1] = fma(r, q.v[4], a[1]);
          });
      if (!G.reduce<2>(L, a, 3, [&](const double (&o)[2]) {
            loop_finish(L, norm0, tol, thr, maxit, timestep, o[0], o[1]);
          }))
        break;
    }
    if (L.done) break;
    const double be = L.beta;
    const bool rst = L.restart != 0;
    loop_cells(
        lo, hi, [&](long long row) { return LoopVals<3>{{r1[row], ap[row], p1[row]}}; },
        [&](long long row, const LoopVals<3> &q) {
          p1[row] = rst ? q.v[0] : fma(be, fma(-w, q.v[1], q.v[2]), q.v[0]);
          if (rst) r0[row] = q.v[0];
        });
    if (!G.sync(L)) break;
  }
  loop_end(L, G);
}

// CG's stop test and beta (finish_cg64) on the loop's scalars (warp 0)
__device__ __forceinline__ void loop_finish_cg(LoopScal &L, double norm0, double tol, int maxit, double n2) {
  double relres, beta, unused;
  div3(sqrt(n2), norm0, n2, L.rho, n2, L.rho, relres, beta, unused);
  if (threadIdx.x != 0) return;
  L.relres = relres;
  if (relres < tol) {
    L.done = 1;
  } else if (!isfinite(relres)) {
    L.done = 1;
    L.status = CFDGB_ENAN;
  } else if (L.iter >= maxit) {
    L.done = 1;
    L.status = CFDGB_ENOCONV;
  } else {
    L.beta = beta;
    L.rho = n2;
    L.iter += 1;
  }
}

__global__ void __launch_bounds__(kLoopBlock, 1) k64cg_loop(Geo g, Stencil<double> st, KrylovVecs<double> v,
                                                            double *part, SolverScal *sc, int iters, int chunk) {
  __shared__ LoopScal L;
  loop_begin(L, sc);
  if (L.done) return;
  LoopGrid G = loop_grid(sc, part);
  const double norm0 = sc->norm0, tol = sc->tol;
  const int maxit = sc->maxit;
  const long long lo = min(g.ncell, (long long)blockIdx.x * chunk), hi = min(g.ncell, lo + chunk);
  double *x = v.x, *r1 = v.r1, *p1 = v.p1, *q1 = v.ap;
  for (int it = 0; it < iters; ++it) {
    {  // q = A p, alpha
      double a[1] = {0.0};
      loop_cells(
          lo, hi, [&](long long row) { return loop_load<0>(g, p1, nullptr, row); },
          [&](long long row, const LoopStencil &S) {
            const double y = loop_apply<0>(g, st, S);
            q1[row] = y;
            a[0] = fma(y, S.c, a[0]);
          });
      if (!G.reduce<1>(L, a, 0, [&](const double (&o)[1]) {
            const double al = L.rho / o[0];
            if (threadIdx.x == 0) L.alpha = al;
          }))
        break;
    }
    const double al = L.alpha;
    {  // x, r, stop test and beta
      double a[1] = {0.0};
      loop_cells(
          lo, hi, [&](long long row) { return LoopVals<4>{{p1[row], q1[row], x[row], r1[row]}}; },
          [&](long long row, const LoopVals<4> &q) {
            x[row] = fma(al, q.v[0], q.v[2]);
            const double r = fma(-al, q.v[1], q.v[3]);
            r1[row] = r;
            a[0] = fma(r, r, a[0]);
          });
      if (!G.reduce<1>(L, a, 1, [&](const double (&o)[1]) { loop_finish_cg(L, norm0, tol, maxit, o[0]); })) break;
    }
    if (L.done) break;
    const double be = L.beta;
    loop_cells(
        lo, hi, [&](long long row) { return LoopVals<2>{{p1[row], r1[row]}}; },
        [&](long long row, const LoopVals<2> &q) { p1[row] = fma(be, q.v[0], q.v[1]); });
    if (!G.sync(L)) break;
  }
  loop_end(L, G);
}

// ---- FP32 CG sweeps in one cooperative launch, the state on chip ----
// A block a multiprocessor keeps a contiguous range of cells for the whole chunk of iterations:
// r and A p in registers, p in shared memory with the plane of cells before and after the range, x in
// shared memory.  What the blocks exchange is r on the cells within a plane of a range's ends
// (through L2): p there is formed again from it by every block that needs it.  So an iteration
// has two grid barriers, both of them reductions, and moves a few megabytes instead of the ten
// vector passes of k32cg*_pq and k32cg_xr.  Same operations per cell as those; the dot products
// are summed in this partition's order.  A thread owns quads of cells along k where nz is a
// multiple of four (V = 4), else single cells.  256x128x64: 21.5 -> 12.1 us an iteration (5.3 of
// it the two reductions; 512 threads with x in registers as well: 12.3).
constexpr int kCgLoopBlock = 1024;
constexpr int kCgLoopCells = 16;                // cells a thread
constexpr size_t kCgLoopShared = 224 * 1024;    // bytes

template <int V>
struct Cells {
  float v[V];
};
template <int V>
__device__ __forceinline__ Cells<V> cells_ld(const float *p) {
  Cells<V> c;
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    c.v[0] = t.x;
    c.v[1] = t.y;
    c.v[2] = t.z;
    c.v[3] = t.w;
  } else {
    c.v[0] = *p;
  }
  return c;
}
template <int V>
__device__ __forceinline__ Cells<V> cells_ldcg(const float *p) {
  Cells<V> c;
  if constexpr (V == 4) {
    const float4 t = __ldcg(reinterpret_cast<const float4 *>(p));
    c.v[0] = t.x;
    c.v[1] = t.y;
    c.v[2] = t.z;
    c.v[3] = t.w;
  } else {
    c.v[0] = __ldcg(p);
  }
  return c;
}
template <int V>
__device__ __forceinline__ void cells_st(float *p, const Cells<V> &c) {
  if constexpr (V == 4)
    *reinterpret_cast<float4 *>(p) = make_float4(c.v[0], c.v[1], c.v[2], c.v[3]);
  else
    *p = c.v[0];
}

// finish_cg32 on the loop's scalars (warp 0)
__device__ __forceinline__ void loop_finish_cg32(LoopScal &L, double norm0, double tol, double delta, int maxit,
                                                 double n2) {
  const double rn = sqrt(n2);
  double relres, beta, unused;
  div3(rn, norm0, n2, L.rho, n2, L.rho, relres, beta, unused);
  if (threadIdx.x != 0) return;
  L.relres = relres;
  if (relres < L.best) L.best = relres;
  if (!isfinite(relres)) {
    L.done = 1;
    L.status = CFDGB_ENAN;
  } else if (L.iter > 16 && relres > 1e3 * L.best) {
    L.done = 1;
    L.status = CFDGB_ENOCONV;
  } else if (L.iter >= maxit) {
    L.done = 1;
    L.status = CFDGB_ENOCONV;
    L.iter += 1;
  } else if (relres < tol || rn < delta * L.rmax) {
    L.done = 1;
    L.status = kStatusRefine;
    L.iter += 1;
  } else {
    L.beta = beta;
    L.rho = n2;
    L.restart = isfinite(beta) ? 0 : 1;
    L.rmax = fmax(L.rmax, rn);
    L.iter += 1;
  }
}

template <int V, int K>
__global__ void __launch_bounds__(kCgLoopBlock, 1) k32cg_loop(Geo g, Stencil<float> st, Vec32 v, double *part,
                                                              SolverScal *sc, int iters, int chunk) {
  extern __shared__ __align__(16) float csm[];
  __shared__ LoopScal L;
  loop_begin(L, sc);
  if (L.done) return;  // the same in every block: sc is written only after the last barrier
  LoopGrid G = loop_grid(sc, part);
  const double norm0 = sc->norm0, tol = sc->tol, delta = sc->delta;
  const int maxit = sc->maxit, tid = threadIdx.x;
  const int n = (int)g.ncell, nz = g.nzc, H = g.nyc * nz;  // a plane
  const int lo = min(n, (int)blockIdx.x * chunk), m = min(n - lo, chunk);
  float *const ps = csm + H;                // p of the range's cells; the planes beside it at -H and m
  float *const xs = csm + 2 * H + chunk;
  const float *const r1 = v.r1;
  float *const pg = sc->par ? v.p[1] : v.p[0];
  const float *const c = st.c[13];  // uniform grid, SPE rows: an axis's coefficient where the neighbour exists
  const float c0 = c[0], c1 = c[1], c2 = c[2], c4 = c[4], c5 = c[5], c6 = c[6];
  // halo cells: h < H before the range, then after it
  const int left = min(lo, H), right = min(n - (lo + m), H);
  Cells<V> r[K], q[K];
  unsigned fl[(K + 3) / 4];  // 8 bits a group: neighbours -x, -y, -z, +z, +y, +x; -z, +z across the wrap
#pragma unroll
  for (int u = 0; u < (K + 3) / 4; ++u) fl[u] = 0;
#pragma unroll
  for (int u = 0; u < K; ++u) {
    const int b = V * (tid + kCgLoopBlock * u);
    if (b >= m) break;
    r[u] = cells_ldcg<V>(r1 + lo + b);
    cells_st<V>(ps + b, cells_ldcg<V>(pg + lo + b));
    cells_st<V>(xs + b, cells_ldcg<V>(v.x + lo + b));
    int ic, jc, kc;
    row_cijk(lo + b, g.nyc, nz, ic, jc, kc);
    const bool pz = g.pz != 0, first = kc == 0, last = kc + V >= nz;
    const unsigned f = (ic > 0) | (jc > 0) << 1 | (!first || pz) << 2 | (!last || pz) << 3 | (jc < g.nyc - 1) << 4 |
                       (ic < g.nxc - 1) << 5 | (first && pz) << 6 | (last && pz) << 7;
    fl[u / 4] |= f << (8 * (u % 4));
  }
  // (a cell beside the range is one thread's, here and in every iteration: no barrier in between)
  for (int h = V * tid; h < left; h += V * kCgLoopBlock) cells_st<V>(ps - left + h, cells_ldcg<V>(pg + lo - left + h));
  for (int h = V * tid; h < right; h += V * kCgLoopBlock) cells_st<V>(ps + m + h, cells_ldcg<V>(pg + lo + m + h));
  for (int it = 0; it < iters; ++it) {
    const float be = (float)L.beta;
    const bool rst = L.restart != 0;
    auto next = [&](float *p, const Cells<V> &rr) {  // p = r + beta p (restart: r)
      Cells<V> t = rr;
      if (!rst) {
        const Cells<V> o = cells_ld<V>(p);
#pragma unroll
        for (int e = 0; e < V; ++e) t.v[e] = fmaf(be, o.v[e], rr.v[e]);
      }
      cells_st<V>(p, t);
    };
#pragma unroll 4
    for (int h = V * tid; h < left; h += V * kCgLoopBlock) next(ps - left + h, cells_ldcg<V>(r1 + lo - left + h));
#pragma unroll 4
    for (int h = V * tid; h < right; h += V * kCgLoopBlock) next(ps + m + h, cells_ldcg<V>(r1 + lo + m + h));
#pragma unroll
    for (int u = 0; u < K; ++u) {
      const int b = V * (tid + kCgLoopBlock * u);
      if (b >= m) break;
      next(ps + b, r[u]);
    }
    __syncthreads();
    float a = 0.0f;
    double a8 = 0.0;
#pragma unroll
    for (int u = 0; u < K; ++u) {  // q = A p: stencil_apply_diff's terms in its order
      const int b = V * (tid + kCgLoopBlock * u);
      if (b >= m) break;
      const unsigned f = fl[u / 4] >> (8 * (u % 4));
      const Cells<V> p = cells_ld<V>(ps + b);
      Cells<V> xm = p, ym = p, yp = p, xp = p;  // a missing neighbour: no difference
      if (f & 1u) xm = cells_ld<V>(ps + b - H);
      if (f & 2u) ym = cells_ld<V>(ps + b - nz);
      if (f & 16u) yp = cells_ld<V>(ps + b + nz);
      if (f & 32u) xp = cells_ld<V>(ps + b + H);
      float zm = p.v[0], zp = p.v[V - 1];
      if (f & 4u) zm = ps[b + ((f & 64u) ? nz - 1 : -1)];
      if (f & 8u) zp = ps[b + ((f & 128u) ? V - nz : V)];
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const float fc = p.v[e];
        float t = c0 * (xm.v[e] - fc);
        t = fmaf(c1, ym.v[e] - fc, t);
        t = fmaf(c2, (e == 0 ? zm : p.v[e > 0 ? e - 1 : 0]) - fc, t);
        t = fmaf(c4, (e == V - 1 ? zp : p.v[e < V - 1 ? e + 1 : V - 1]) - fc, t);
        t = fmaf(c5, yp.v[e] - fc, t);
        t = fmaf(c6, xp.v[e] - fc, t);
        q[u].v[e] = t;
        a = fmaf(t, fc, a);
      }
      if (V == 1 && u % 8 == 7) {  // FP32 runs of eight products, as k32cg_pq's (AccF)
        a8 += (double)a;
        a = 0.0f;
      }
    }
    {
      double d[1] = {a8 + (double)a};
      if (!G.reduce<1>(L, d, 0, [&](const double (&o)[1]) {
            const double al = L.rho / o[0];
            if (threadIdx.x == 0) L.alpha = al;
          }))
        break;
    }
    const float al = (float)L.alpha;
    a = 0.0f;
#pragma unroll
    for (int u = 0; u < K; ++u) {
      const int b = V * (tid + kCgLoopBlock * u);
      if (b >= m) break;
      const Cells<V> p = cells_ld<V>(ps + b);
      Cells<V> x = cells_ld<V>(xs + b);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        x.v[e] = fmaf(al, p.v[e], x.v[e]);
        r[u].v[e] = fmaf(-al, q[u].v[e], r[u].v[e]);
        a = fmaf(r[u].v[e], r[u].v[e], a);
      }
      cells_st<V>(xs + b, x);
      if (b < H || b >= m - H) cells_st<V>(v.r1 + lo + b, r[u]);  // what other blocks read
    }
    {
      double d[1] = {(double)a};
      if (!G.reduce<1>(L, d, 1, [&](const double (&o)[1]) { loop_finish_cg32(L, norm0, tol, delta, maxit, o[0]); })) break;
    }
    if (L.done) break;
  }
#pragma unroll
  for (int u = 0; u < K; ++u) {
    const int b = V * (tid + kCgLoopBlock * u);
    if (b >= m) break;
    cells_st<V>(v.r1 + lo + b, r[u]);
    cells_st<V>(v.x + lo + b, cells_ld<V>(xs + b));
    cells_st<V>(pg + lo + b, cells_ld<V>(ps + b));
  }
  loop_end(L, G);
}

// The neighbours of a cell in the order of stencil_apply's terms: -x, -y, -z, +z, +y, +x
// (row -1 where there is none) and the row's coefficients
struct LoopRow {
  int nb[6];
  double c[7];
};
__device__ __forceinline__ LoopRow loop_row(const Geo &g, const Stencil<double> &st, int row) {
  LoopRow R;
  int ic, jc, kc;
  row_cijk(row, g.nyc, g.nzc, ic, jc, kc);
  const int nyz = g.nyc * g.nzc;
  R.nb[0] = ic > 0 ? row - nyz : -1;
  R.nb[1] = jc > 0 ? row - g.nzc : -1;
  R.nb[2] = (int)z_minus(g, kc, row);
  R.nb[3] = (int)z_plus(g, kc, row);
  R.nb[4] = jc < g.nyc - 1 ? row + g.nzc : -1;
  R.nb[5] = ic < g.nxc - 1 ? row + nyz : -1;
#pragma unroll
  for (int q = 0; q < 7; ++q)
    R.c[q] = g.nonuni ? g.cof[st.jac][q * g.ncell + row] : st.c[cls_of(g, ic, jc, kc)][q];
  return R;
}
// A f from the centre and the neighbours' values (zero where there is none)
__device__ __forceinline__ double loop_row_apply(const LoopRow &R, const double (&f)[6], double fc) {
  double y = R.c[0] * f[0];
  y = fma(R.c[1], f[1], y);
  y = fma(R.c[2], f[2], y);
  y = fma(R.c[3], fc, y);
  y = fma(R.c[4], f[3], y);
  y = fma(R.c[5], f[4], y);
  return fma(R.c[6], f[5], y);
}

// One cell a thread (grids up to the device's threads in this form): the thread's own values
// stay in registers for the whole chunk, and p and s are also formed at the six neighbours from
// the published r1 and A p, so that an iteration has three barriers instead of five.
__global__ void __launch_bounds__(kLoopBlock, 1) k64_bicg_loop1(Geo g, Stencil<double> st, KrylovVecs<double> v,
                                                                double *part, SolverScal *sc, int iters, int chunk) {
  __shared__ LoopScal L;
  loop_begin(L, sc);
  if (L.done) return;
  LoopGrid G = loop_grid(sc, part);
  const double norm0 = sc->norm0, tol = sc->tol, thr = sc->restart_thr;
  const int maxit = sc->maxit, timestep = sc->timestep;
  const int row = blockIdx.x * chunk + threadIdx.x;
  const bool on = (int)threadIdx.x < chunk && row < g.ncell;
  LoopRow R{};
  double x = 0, r0 = 0, r1 = 0, p = 0, ap = 0;
  double rn[6] = {0, 0, 0, 0, 0, 0}, pn[6] = {0, 0, 0, 0, 0, 0};  // r1 and p at the neighbours
  if (on) {
    R = loop_row(g, st, row);
    x = v.x[row];
    r0 = v.r0[row];
    r1 = v.r1[row];
    p = v.p1[row];
#pragma unroll
    for (int q = 0; q < 6; ++q)
      if (R.nb[q] >= 0) {
        rn[q] = v.r1[R.nb[q]];
        pn[q] = v.p1[R.nb[q]];
      }
  }
  for (int it = 0; it < iters; ++it) {
    {  // A p, published (its neighbours read the last one two barriers ago)
      double a[1] = {0.0};
      if (on) {
        ap = loop_row_apply(R, pn, p);
        v.ap[row] = ap;
        a[0] = ap * r0;
      }
      if (!G.reduce<1>(L, a, 0, [&](const double (&o)[1]) {
            const double al = L.rho / o[0];
            if (threadIdx.x == 0) L.alpha = al;
          }))
        break;
    }
    const double al = L.alpha;
    double sv = 0, as = 0, an[6] = {0, 0, 0, 0, 0, 0};
    {
      double a[2] = {0.0, 0.0};
      if (on) {
        double sn[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) an[q] = R.nb[q] >= 0 ? __ldcg(v.ap + R.nb[q]) : 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) sn[q] = fma(-al, an[q], rn[q]);
        sv = fma(-al, ap, r1);
        as = loop_row_apply(R, sn, sv);
        a[0] = as * sv;
        a[1] = as * as;
      }
      if (!G.reduce<2>(L, a, 1, [&](const double (&o)[2]) {
            const double w = o[0] / o[1];
            if (threadIdx.x == 0) L.omega = w;
          }))
        break;
    }
    const double w = L.omega;
    {
      double a[2] = {0.0, 0.0};
      if (on) {
        x = fma(w, sv, fma(al, p, x));
        r1 = fma(-w, as, sv);
        v.r1[row] = r1;  // published: its neighbours read the last one two barriers ago
        a[0] = r1 * r1;
        a[1] = r1 * r0;
      }
      if (!G.reduce<2>(L, a, 3, [&](const double (&o)[2]) {
            loop_finish(L, norm0, tol, thr, maxit, timestep, o[0], o[1]);
          }))
        break;
    }
    if (L.done) break;
    const double be = L.beta;
    const bool rst = L.restart != 0;
    if (on) {  // p here and at the neighbours
      p = rst ? r1 : fma(be, fma(-w, ap, p), r1);
      if (rst) r0 = r1;
#pragma unroll
      for (int q = 0; q < 6; ++q)
        if (R.nb[q] >= 0) {
          rn[q] = __ldcg(v.r1 + R.nb[q]);
          pn[q] = rst ? rn[q] : fma(be, fma(-w, an[q], pn[q]), rn[q]);
        }
    }
  }
  if (on) {
    v.x[row] = x;
    v.r0[row] = r0;
    v.p1[row] = p;
  }
  loop_end(L, G);
}

// bicgstabRe2.hpp:133-153: at the cap, NaN/Inf entries come from the previous solution;
// if more than 10 % were bad, the whole vector comes from the one before.
__global__ void __launch_bounds__(kBlock) k_nan_replace(Geo g, double *x, const double *px1, double *part,
                                                        SolverScal *sc) {
  if (sc->status != CFDGB_ENOCONV) return;
  double bad[1] = {0.0}, out[1];
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double xv = x[row];
    if (isnan(xv) || isinf(xv)) { x[row] = px1[row]; bad[0] += 1.0; }
  }
  if (grid_sum<1>(bad, part, &sc->cnt[4], out) && lin_tid() == 0)
    sc->restart = out[0] > (double)g.ncell * 0.1 ? 2 : 0;
}
__global__ void __launch_bounds__(kBlock) k_nan_restore(Geo g, double *x, const double *px2, const SolverScal *sc) {
  if (sc->status != CFDGB_ENOCONV || sc->restart != 2) return;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    x[row] = px2[row];
  }
}

// ---- mixed precision: FP32 BiCGSTAB inside FP64 iterative refinement ----
// Each sweep runs FP32 BiCGSTAB from a fresh start on r1 = (r - null-space part) / scale
// (scale fixed for the whole solve) until its residual has dropped by delta; its
// correction accumulates in the FP32 x.  The refinement adds scale * x to the FP64
// solution and recomputes r = b - A x in FP64, which starts the next sweep.  Keeping the
// Krylov space across refinements (reliable updates) was measured too: on the 512-cell
// axis the FP32 iteration then breaks down near 1e-3 (with compensated dot products as
// well: the FP32 vectors and stencil are the limit), while short restarted sweeps
// converge to the FP64 tolerance.

// r = b - A x in FP64, stored rounded to FP32 (rf); ||r||, ||b|| (flags & 1) and the sweep
// scale (flags & 2): the power of two at or below ||r||, so that scaling by it, here and in
// k_correct64, is exact.  jacobi: st holds the jp-scaled rows (st.c[.][7] = jp), whose
// unscaled residual is r / jp.  FIRST: also ||b|| (a solve's first residual).  The kernel
// is bound by the FP64 pipe, so only the residual (7 FMA from b) and the norms are FP64; the
// null-space sum (whose only use is to keep the FP32 system consistent) is summed in FP32
// per thread, and is left out on the stretched grid (whose residual is taken as it is).
template <bool FIRST>
__global__ void __launch_bounds__(kBlock) k_residual64(Geo g, Stencil<double> st, int jacobi,
                                                        const double *__restrict__ b, const double *__restrict__ x,
                                                        float *__restrict__ rf, double *part, StepScal *ss,
                                                        SolverScal *inner, int flags) {
  double acc[3] = {0.0, 0.0, 0.0};
  float ns = 0.0f;
  const bool nsum = !g.nonuni;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double bb = b[row];
    const double r = resid_at(g, st, x, ic, jc, kc, row, bb);
    const float r32 = d2f_int(r);
    rf[row] = r32;
    acc[0] += r * r;
    if (FIRST) acc[1] += bb * bb;
    // the unscaled residual's sum: its component along the operator's null space
    if (nsum) ns += jacobi ? r32 * d2f_int(row_diag(g, st, ic, jc, kc, row)) : r32;
  }
  acc[2] = f2d_int(ns);
  double out[3];
  if (grid_sum<3>(acc, part, &ss->cnt[1], out) && lin_tid() == 0) {
    if (flags & 1) ss->bnorm = sqrt(out[1]);
    ss->rnorm = sqrt(out[0]);
    ss->relres = ss->rnorm / ss->bnorm;
    ss->rsum = out[2];
    if (flags & 2) inner->scale = sweep_scale(ss->rnorm);
  }
}

// The same residual on a uniform grid with an even nz, formed from 64-bit integers: at 1/32 of
// the integer pipes' rate the seven FP64 FMAs of a row cost six times its memory traffic.  A thread
// owns two rows of a pair of cells along k and marches along x; z neighbours across pairs by
// shuffles.  It takes the values its four cells need in units of its own, u = 2^(em - 1082) for an
// exponent field em at or above all of theirs (|x| <= 2^60 u, truncated), so the differences
// x_c - x_nb are integers; the row is jp sum_a w_a (2 x_c - x_l - x_r) with w_a = 1/h_a^2 a 60-bit
// integer (30 and 30 bits: the products are twelve wide multiply-adds), converted once and
// subtracted from b in FP64.  em is kept from plane to plane while it covers the values and
// the largest |x| in each cell's stencil, m, is at least 2^-kFixSpan of 2^(em - 1023): then u <= 2^-54
// m, and the error, 4 u w from each of three differences and 4 u w from the sum's rounding, is below
// 2^-50 w m, the FMA chain's being up to seven roundings of 2^-53 of its partial sums, 12 w m.  (In
// one unit for the whole grid, taken from its largest |x|, quiet regions kept fewer bits than
// FP64: 73 us, but errors of 1e10 times that bound where x falls over twelve decades.)  Cells that no such em serves (zeros, Inf, NaN, extreme exponents, a peak beside values
// 2^-5 of it) take the FMA chain.  Three FP64-pipe instructions a cell (the conversion, the
// subtraction and the norm).  The next plane's loads are issued before this one's arithmetic.
// 512x256x64: the FMA chain 164 us, this 95 (236 instructions a cell, issue 55 % at 16 warps a
// multiprocessor).
constexpr int kFixSpan = 5;
struct FixOp {
  unsigned wh[3], wl[3];  // 1/h^2 per axis times 2^k, its parts above and below 2^30
  int k;
  float dg[27];           // the unscaled diagonal per class, rounded to FP32
};

// sum_a w_a s_a in units of 2^62, rounded to nearest (|s_a| <= 2^62, w_a < 2^60).  All four partial
// products a pair (a 2^62 + b 2^32 + c 2^30 + d; three of each fit 64 bits) and one rounding: with the
// lowest left out and the others truncated the sum lost up to five units, all of one sign.
__device__ __forceinline__ long long fix_dot(const FixOp &F, long long sx, long long sy, long long sz) {
  const int hx = (int)(sx >> 32), hy = (int)(sy >> 32), hz = (int)(sz >> 32);
  const unsigned lx = (unsigned)sx, ly = (unsigned)sy, lz = (unsigned)sz;
  long long a = (long long)hx * (int)F.wh[0], b = (long long)hx * (int)F.wl[0];
  unsigned long long c = (unsigned long long)lx * F.wh[0], d = (unsigned long long)lx * F.wl[0];
  a += (long long)hy * (int)F.wh[1];
  b += (long long)hy * (int)F.wl[1];
  c += (unsigned long long)ly * F.wh[1];
  d += (unsigned long long)ly * F.wl[1];
  a += (long long)hz * (int)F.wh[2];
  b += (long long)hz * (int)F.wl[2];
  c += (unsigned long long)lz * F.wh[2];
  d += (unsigned long long)lz * F.wl[2];
  c += (d >> 30) + ((unsigned long long)((unsigned)b & 0x3fffffffu) << 2) + 0x80000000ULL;
  return a + (b >> 30) + (long long)(c >> 32);
}

template <bool FIRST>
__global__ void __launch_bounds__(kBlock, 2) k_residual_fx(Geo g, Stencil<double> st, FixOp F, int jacobi,
                                                            const double *__restrict__ b, const double *__restrict__ x,
                                                            float *__restrict__ rf, double *part, StepScal *ss,
                                                            SolverScal *inner, int flags) {
  const int W = blockDim.x, lane = threadIdx.x, nz = g.nzc;  // W pairs of a row, a power of two up to a warp
  const int kc = 2 * (blockIdx.x * W + lane), jc = 2 * (blockIdx.y * blockDim.y + threadIdx.y);
  const bool on = kc < nz && jc < g.nyc, on1 = on && jc + 1 < g.nyc;
  const int chunk = (g.nxc + gridDim.z - 1) / gridDim.z;
  const int i0 = min(g.nxc, (int)blockIdx.z * chunk), i1 = min(g.nxc, i0 + chunk);
  const int nyz = g.nyc * nz;
  const bool whole = nz == 2 * W;                      // a row is one segment of lanes
  const bool zl = kc > 0 || g.pz, zr = kc + 2 < nz || g.pz;  // cells left and right of the pair exist
  const bool sl = whole || lane > 0, sr = whole || (lane + 1 < W && kc + 2 < nz);  // and come by shuffle
  const int wl = kc > 0 ? -1 : nz - 1, wr = kc + 2 < nz ? 2 : 2 - nz;
  // classes of the four cells, less the plane's part
  const int cy0 = 3 * axis_class(jc, g.nyc), cy1 = 3 * axis_class(jc + 1, g.nyc);
  const int cz0 = g.pz ? 1 : axis_class(kc, nz), cz1 = g.pz ? 1 : axis_class(kc + 1, nz);
  double acc[3] = {0.0, 0.0, 0.0};
  float ns = 0.0f;
  // a row's pair of residuals, stored; and from A x (y0, y1)
  auto put = [&](long long row, int c0, int c1, double r0, double r1, double2 bb) {
    const float f0 = d2f_int(r0), f1 = d2f_int(r1);
    *reinterpret_cast<float2 *>(rf + row) = make_float2(f0, f1);
    acc[0] = fma(r0, r0, acc[0]);
    acc[0] = fma(r1, r1, acc[0]);
    if (FIRST) {
      acc[1] = fma(bb.x, bb.x, acc[1]);
      acc[1] = fma(bb.y, bb.y, acc[1]);
    }
    // the unscaled residual's sum: its component along the operator's null space
    ns += jacobi ? fmaf(f0, F.dg[c0], f1 * F.dg[c1]) : f0 + f1;
  };
  auto finish = [&](long long row, int c0, int c1, double y0, double y1, double2 bb) {
    put(row, c0, c1, jacobi ? fma(-st.c[c0][7], y0, bb.x) : bb.x - y0,
        jacobi ? fma(-st.c[c1][7], y1, bb.y) : bb.y - y1, bb);
  };
  long long row = ((long long)i0 * g.nyc + jc) * nz + kc;
  struct Pair {
    long long a, b;
  };
  auto size = [](double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; };  // ordered as |v|
  auto largest = [&](double2 p, double2 q) { return max(max(size(p.x), size(p.y)), max(size(q.x), size(q.y))); };
  double2 x0, x1;                                // the two rows' cells
  Pair c0{0, 0}, c1{0, 0}, dm0{0, 0}, dm1{0, 0};  // in units of em, and their differences to the plane before
  int em = 0;                                    // 0: none
  // the loads a plane needs, issued a plane ahead: both rows of the next plane, the rows below
  // and above, b of both rows
  double2 np0, np1, nlo, nhi, nb0, nb1;
  x0 = x1 = np0 = np1 = nlo = nhi = nb0 = nb1 = make_double2(0.0, 0.0);
  auto ahead = [&](int ic, long long r) {
    if (!on || ic >= i1) return;
    nb0 = *reinterpret_cast<const double2 *>(b + r);
    if (on1) nb1 = *reinterpret_cast<const double2 *>(b + r + nz);
    if (ic + 1 < g.nxc) {
      np0 = *reinterpret_cast<const double2 *>(x + r + nyz);
      if (on1) np1 = *reinterpret_cast<const double2 *>(x + r + nz + nyz);
    }
    if (jc > 0) nlo = *reinterpret_cast<const double2 *>(x + r - nz);
    if (jc + 2 < g.nyc) nhi = *reinterpret_cast<const double2 *>(x + r + 2 * nz);
  };
  auto fix = [&](double2 v) { return Pair{d2fix(v.x, em), d2fix(v.y, em)}; };
  ahead(i0, row);
  if (on && i0 < i1) {
    x0 = *reinterpret_cast<const double2 *>(x + row);
    x1 = on1 ? *reinterpret_cast<const double2 *>(x + row + nz) : x0;
  }
  for (int ic = i0; ic < i1; ++ic, row += nyz) {
    double2 q0 = x0, q1 = x1, lo = x0, hi = x1;  // next plane; rows below and above: a missing one has no difference
    const double2 b0 = nb0, b1 = nb1;
    if (on) {
      if (ic + 1 < g.nxc) {
        q0 = np0;
        q1 = on1 ? np1 : np0;
      }
      if (jc > 0) lo = nlo;
      if (jc + 2 < g.nyc) hi = nhi;
    }
    ahead(ic + 1, row + nyz);
    const int lf = (lane - 1) & (W - 1), rt = (lane + 1) & (W - 1);
    double l0 = __shfl_sync(0xffffffffu, x0.y, lf, W), r0 = __shfl_sync(0xffffffffu, x0.x, rt, W);
    double l1 = __shfl_sync(0xffffffffu, x1.y, lf, W), r1 = __shfl_sync(0xffffffffu, x1.x, rt, W);
    if (on) {
      if (!zl) {
        l0 = x0.x;
        l1 = x1.x;
      } else if (!sl) {
        l0 = x[row + wl];
        l1 = on1 ? x[row + nz + wl] : l0;
      }
      if (!zr) {
        r0 = x0.y;
        r1 = x1.y;
      } else if (!sr) {
        r0 = x[row + wr];
        r1 = on1 ? x[row + nz + wr] : r0;
      }
      // the largest value, and a lower bound of each cell's: every one of the four stencils holds
      // three of the four cells, so the second largest of them
      const unsigned top = max(max(largest(x0, x1), largest(q0, q1)),
                               max(largest(lo, hi), largest(make_double2(l0, l1), make_double2(r0, r1))));
      const unsigned sa = size(x0.x), sb = size(x0.y), sc = size(x1.x), sd = size(x1.y);
      const int least = (int)(max(min(max(sa, sb), max(sc, sd)), max(min(sa, sb), min(sc, sd))) >> 20);
      if ((int)(top >> 20) > em || least + kFixSpan < em) {  // (rare: the values drift by powers of two)
        double2 m0 = x0, m1 = x1;
        if (ic > 0) {
          m0 = *reinterpret_cast<const double2 *>(x + row - nyz);
          m1 = on1 ? *reinterpret_cast<const double2 *>(x + row + nz - nyz) : m0;
        }
        em = (int)(max(top, largest(m0, m1)) >> 20) + 1;  // room for a factor of two
        if (least + kFixSpan < em) --em;
        if (least + kFixSpan < em || em < 200 || em > 1900) em = 0;
        if (em) {
          c0 = fix(x0);
          c1 = fix(x1);
          const Pair f0 = fix(m0), f1 = fix(m1);
          dm0 = Pair{c0.a - f0.a, c0.b - f0.b};
          dm1 = Pair{c1.a - f1.a, c1.b - f1.b};
        }
      }
      const int cx = 9 * axis_class(ic, g.nxc);
      if (em) {
        const int shift = 62 - F.k - 1082 + em;
        const Pair p0 = fix(q0), p1 = fix(q1), lw = fix(lo), up = fix(hi);
        const Pair dp0{p0.a - c0.a, p0.b - c0.b};
        const Pair dy{on1 ? c1.a - c0.a : 0, on1 ? c1.b - c0.b : 0};  // row 1 less row 0
        const long long dz0 = c0.b - c0.a;
        const double y0 = fix2d(fix_dot(F, dm0.a - dp0.a, (c0.a - lw.a) - dy.a, (c0.a - d2fix(l0, em)) - dz0), shift);
        const double y1 = fix2d(fix_dot(F, dm0.b - dp0.b, (c0.b - lw.b) - dy.b, dz0 - (d2fix(r0, em) - c0.b)), shift);
        finish(row, cx + cy0 + cz0, cx + cy0 + cz1, y0, y1, b0);
        dm0 = dp0;
        if (on1) {
          const Pair dp1{p1.a - c1.a, p1.b - c1.b};
          const long long dz1 = c1.b - c1.a;
          const double y2 = fix2d(fix_dot(F, dm1.a - dp1.a, dy.a - (up.a - c1.a), (c1.a - d2fix(l1, em)) - dz1), shift);
          const double y3 = fix2d(fix_dot(F, dm1.b - dp1.b, dy.b - (up.b - c1.b), dz1 - (d2fix(r1, em) - c1.b)), shift);
          finish(row + nz, cx + cy1 + cz0, cx + cy1 + cz1, y2, y3, b1);
          dm1 = dp1;
        }
        c0 = p0;
        c1 = p1;
      } else {
        for (int e = 0; e < (on1 ? 2 : 1); ++e) {
          const long long r = row + (long long)e * nz;
          const double2 bb = e ? b1 : b0;
          const int c = cx + (e ? cy1 : cy0);
          put(r, c + cz0, c + cz1, resid_at(g, st, x, ic, jc + e, kc, r, bb.x),
              resid_at(g, st, x, ic, jc + e, kc + 1, r + 1, bb.y), bb);
        }
      }
    }
    x0 = q0;
    x1 = q1;
  }
  acc[2] = f2d_int(ns);
  double out[3];
  if (grid_sum<3>(acc, part, &ss->cnt[1], out) && lin_tid() == 0) {
    if (flags & 1) ss->bnorm = sqrt(out[1]);
    ss->rnorm = sqrt(out[0]);
    ss->relres = ss->rnorm / ss->bnorm;
    ss->rsum = out[2];
    if (flags & 2) inner->scale = sweep_scale(ss->rnorm);
  }
}

// rf minus its null-space part (the mean of the unscaled residual; for the Jacobi rows its
// image jp * mean), divided by the sweep scale, in FP32 (the division by a power of two is
// exact).  Removing it keeps the FP32 system consistent, so the iteration cannot drift
// along the constant mode.
__device__ __forceinline__ float scaled_residual(const Geo &g, const Stencil<double> &st, int jacobi,
                                                 const float *__restrict__ rf, float mi, float inv, int ic, int jc,
                                                 int kc, long long row) {
  const float r = rf[row] * inv;
  return jacobi ? fmaf(-mi, d2f_int(row_jp(g, st, ic, jc, kc, row)), r) : r - mi;
}

// start of a sweep: x = 0, r1 = scaled residual, rho = <r1, r1>; restart = 1 makes the first p
// kernel set r0 = r1 and take p = r1 (the reference's p1 = r0); delta, peak: this sweep's
// residual reductions (against its start and its largest residual).  first: also the solve's
// set-up (iteration count, the FP32 estimate's normalisation).
__global__ void __launch_bounds__(kBlock) k_refine_start32(Geo g, Stencil<double> st, int jacobi, Vec32 v,
                                                            const float *__restrict__ rf, const StepScal *ss,
                                                            double delta, double peak, int first, double *part,
                                                            SolverScal *sc) {
  const double inv = sc->scale > 0.0 ? 1.0 / sc->scale : 0.0;  // a power of two
  // the null-space part is the mean on the uniform grid (a symmetric operator); on the
  // stretched grid the operator's left null vector is not constant, and the FP64 residual,
  // in range(A) for a consistent system, is taken as it is
  const double m = g.nonuni ? 0.0 : ss->rsum / (double)g.ncell;
  const float inv32 = d2f_int(inv), mi = d2f_int(m * inv);
  Dot2F acc;
  FOR_CELLS4(g) {
    const long long row = ROW(g);
    const float r = scaled_residual(g, st, jacobi, rf, mi, inv32, ic, jc, kc, row);
    v.x[row] = 0.0f;
    v.r1[row] = r;
    acc.add(r, r);
  }
  double a[1] = {acc.get()}, out[1];
  if (grid_sum<1>(a, part, &sc->cnt[0], out) && lin_tid() == 0) {
    if (first) {
      sc->fault = 0;
      sc->timestep += 1;
      sc->norm0 = ss->bnorm * inv;  // relres = ||r1|| scale / ||b||
      sc->best = ss->relres;
      sc->iter = 0;
    }
    sc->delta = delta;
    sc->peak = peak;
    sc->rho = out[0];
    sc->rmax = sqrt(out[0]);
    sc->rstart = sc->rmax;
    sc->relres = sqrt(out[0]) / sc->norm0;
    sc->rel0 = sc->relres;
    sc->snap_rel = sc->relres;  // x = 0, kept by the first x update
    sc->snap = 1;
    sc->snap_iter = sc->iter;
    sc->stall = max(kSweepStall, 2 * (g.nxc + g.nyc + g.nzc));
    sc->done = 0;
    sc->status = 0;
    sc->restart = 1;
    sc->par = 0;
  }
}

// sum of e: FP32 per thread (its only use is the constant mode, which the operator
// annihilates, so its rounding changes x by a constant), FP64 over threads.  Pointwise on
// the compact vector: quads over a flat grid-stride loop (g.xgrid blocks), the tail cells
// of a cell count that is not a multiple of 4 by the first threads.
__global__ void __launch_bounds__(kBlock) k_sum32(Geo g, const float *__restrict__ e, double *part, StepScal *ss) {
  float f = 0.0f;
  const long long nq = g.ncell / 4, stride = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long q = t0; q < nq; q += stride) {
    const float4 v = *reinterpret_cast<const float4 *>(e + 4 * q);
    f += (v.x + v.y) + (v.z + v.w);
  }
  if (t0 < g.ncell - 4 * nq) f += e[4 * nq + t0];
  double acc[1] = {f2d_int(f)};
  double out[1];
  if (grid_sum<1>(acc, part, &ss->cnt[5], out) && lin_tid() == 0) ss->esum = out[0];
}

// x += factor (e - mean e): factor = +-2^k, the sweep scale, applies an inner correction
// (+) or takes it back (-); the mean (the constant mode, which the pressure leaves free) is
// dropped.  e - mean in FP32, widened exactly, scaled by 2^k and signed in its bits: one
// FP64 addition a cell.  Pointwise, quads as k_sum32.
__device__ __forceinline__ double correction(float e, float m, long long shift, long long sign) {
  const float f = e - m;
  const long long d = __double_as_longlong(f2d_int(f));
  // a zero stays zero (tested in FP32: the test of d is one of the FP64 pipe's); any other
  // value is an FP32 normal, far from the FP64 limits
  return __longlong_as_double((__float_as_uint(f) & 0x7f800000u) == 0u ? 0LL : (d + shift) ^ sign);
}
__global__ void __launch_bounds__(kBlock) k_correct64(Geo g, double *__restrict__ x, const float *__restrict__ e,
                                                       int k, int neg, const StepScal *ss) {
  const float m = d2f_int(ss->esum / (double)g.ncell);
  const long long shift = (long long)k << 52, sign = neg ? (long long)0x8000000000000000ULL : 0LL;
  const long long nq = g.ncell / 4, stride = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long q = t0; q < nq; q += stride) {
    const float4 v = *reinterpret_cast<const float4 *>(e + 4 * q);
    double2 *xp = reinterpret_cast<double2 *>(x + 4 * q);
    double2 a = xp[0], b = xp[1];
    a.x += correction(v.x, m, shift, sign);
    a.y += correction(v.y, m, shift, sign);
    b.x += correction(v.z, m, shift, sign);
    b.y += correction(v.w, m, shift, sign);
    xp[0] = a;
    xp[1] = b;
  }
  if (t0 < g.ncell - 4 * nq) x[4 * nq + t0] += correction(e[4 * nq + t0], m, shift, sign);
}

// ---- null-space projection of the right-hand side (project_rhs) ----
// The Neumann operator annihilates constants, so b must sum to zero (unscaled rows) for
// the system to have a solution.  rsum = sum of the unscaled b; b -= its mean, mapped
// back through jp for the Jacobi rows.
__global__ void __launch_bounds__(kBlock) k_rhs_sum(Geo g, Stencil<double> st, int jacobi,
                                                     const double *__restrict__ b, double *part, StepScal *ss) {
  double acc[1] = {0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    acc[0] += jacobi ? b[row] * row_diag(g, st, ic, jc, kc, row) : b[row];
  }
  double out[1];
  if (grid_sum<1>(acc, part, &ss->cnt[6], out) && lin_tid() == 0) ss->rsum = out[0];
}
__global__ void __launch_bounds__(kBlock) k_rhs_subtract(Geo g, Stencil<double> st, int jacobi,
                                                          double *__restrict__ b, const StepScal *ss) {
  const double m = ss->rsum / (double)g.ncell;
  FOR_CELLS(g) {
    const long long row = ROW(g);
    b[row] -= jacobi ? m * row_jp(g, st, ic, jc, kc, row) : m;
  }
}

// out = in scaled to the rows of the system: by jp (Jacobi-scaled rows) or unchanged
__global__ void __launch_bounds__(kBlock) k_scale_rows(Geo g, Stencil<double> st, int jacobi,
                                                        const double *__restrict__ in, double *__restrict__ out) {
  FOR_CELLS(g) {
    const long long row = ROW(g);
    out[row] = jacobi ? row_jp(g, st, ic, jc, kc, row) * in[row] : in[row];
  }
}

// ---- red-black SOR (FP64) on the exact Neumann rows ----
// One colour per launch: cells with (i+j+k) even, then odd, so each half-sweep updates
// cells whose neighbours all have the other colour (no race, order independent; periodic z
// needs an even nzc for the cells across the wrap to differ in colour).
__global__ void __launch_bounds__(kBlock) k_rbsor(Geo g, Stencil<double> st, const double *__restrict__ b,
                                                   double *__restrict__ x, double omega, int color) {
  const long long nyz = (long long)g.nyc * g.nzc;
  FOR_CELLS(g) {
    if (((ic + jc + kc) & 1) != color) continue;
    const long long row = ROW(g);
    const double *c = st.c[cls_of(g, ic, jc, kc)];
    double off = 0.0;
    if (ic > 0) off += c[0] * x[row - nyz];
    if (jc > 0) off += c[1] * x[row - g.nzc];
    const long long zm = z_minus(g, kc, row), zp = z_plus(g, kc, row);
    if (zm >= 0) off += c[2] * x[zm];
    if (zp >= 0) off += c[4] * x[zp];
    if (jc < g.nyc - 1) off += c[5] * x[row + g.nzc];
    if (ic < g.nxc - 1) off += c[6] * x[row + nyz];
    const double xn = (b[row] - off) * c[7];  // c[7] = 1/diag (no division in the sweep)
    x[row] += omega * (xn - x[row]);
  }
}

__global__ void __launch_bounds__(kBlock) k_residual_norm64(Geo g, Stencil<double> st, const double *__restrict__ b,
                                                             const double *__restrict__ x, double *part, StepScal *ss) {
  double acc[1] = {0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    const double r = b[row] - spmv_at<double>(g, st, x, ic, jc, kc, row);
    acc[0] += r * r;
  }
  double out[1];
  if (grid_sum<1>(acc, part, &ss->cnt[2], out) && lin_tid() == 0) {
    ss->rnorm = sqrt(out[0]);
    ss->relres = ss->rnorm / ss->bnorm;
  }
}

__global__ void __launch_bounds__(kBlock) k_vec_norm64(Geo g, const double *__restrict__ b, double *part, StepScal *ss) {
  double acc[1] = {0.0};
  FOR_CELLS(g) {
    const long long row = ROW(g);
    acc[0] += b[row] * b[row];
  }
  double out[1];
  if (grid_sum<1>(acc, part, &ss->cnt[3], out) && lin_tid() == 0) ss->bnorm = sqrt(out[0]);
}

// ---- launchers ----
static inline dim3 cgrid(const Geo &g) { return dim3(g.lgx, g.lgy, g.lgz); }
static inline dim3 cblock(const Geo &g) { return dim3(g.lbx, g.lby, 1); }
static inline Vec32 v32(const KrylovVecs<float> &v, float *const p2[2], float *const ap2[2]) {
  Vec32 o;
  o.x = v.x; o.r0 = v.r0; o.r1 = v.r1; o.s = v.s; o.as = v.as;
  o.p[0] = p2[0]; o.p[1] = p2[1]; o.ap[0] = ap2[0]; o.ap[1] = ap2[1];
  o.xb = v.xb;
  return o;
}

// the stretched grid's rows, [7][ncell]: every column of nonuni_row, zeros included
__global__ void __launch_bounds__(kBlock) k_build_rows(Geo g, int jac, double *__restrict__ out) {
  FOR_CELLS(g) {
    const long long row = ROW(g);
    double c[8];
    nonuni_row(g, jac, ic, jc, kc, row, c);
#pragma unroll
    for (int q = 0; q < 7; ++q) out[q * g.ncell + row] = c[q];
  }
}

void launch_build_rows(cudaStream_t s, const Geo &g, int jac, double *out) {
  k_build_rows<<<cgrid(g), cblock(g), 0, s>>>(g, jac, out);
}

// the stored rows rounded to FP32 (MIXED on the stretched grid)
__global__ void __launch_bounds__(kBlock) k_rows_f32(long long n, const double *__restrict__ in,
                                                     float *__restrict__ out) {
  for (long long q = blockIdx.x * (long long)kBlock + threadIdx.x; q < n; q += (long long)gridDim.x * kBlock)
    out[q] = (float)in[q];
}
void launch_rows_f32(cudaStream_t s, long long n, const double *in, float *out) {
  k_rows_f32<<<(int)std::min<long long>((n + kBlock - 1) / kBlock, 4096), kBlock, 0, s>>>(n, in, out);
}

void launch_bicg_setup64(cudaStream_t s, int, const Geo &g, const Stencil<double> &st, KrylovVecs<double> v,
                         const double *b, double *px1, double *px2, double *part, SolverScal *sc, int restart) {
  k_bicg_setup64<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, b, px1, px2, part, sc, restart);
}

void launch_bicgp64_part(cudaStream_t s, int part, const Geo &g, const Stencil<double> &st, PrecVecsT<double> v,
                         double *part_buf, SolverScal *sc) {
  switch (part) {
    case 0: k64p_p<<<cgrid(g), cblock(g), 0, s>>>(g, v, sc); break;
    case 1: k64p_v<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, part_buf, sc); break;
    case 2: k64p_s<<<cgrid(g), cblock(g), 0, s>>>(g, v, sc); break;
    case 3: k64p_t<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, part_buf, sc); break;
    default: k64p_xr<<<cgrid(g), cblock(g), 0, s>>>(g, v, part_buf, sc); break;
  }
}

void launch_bicg64_part(cudaStream_t s, int part, const Geo &g, const Stencil<double> &st, KrylovVecs<double> v,
                        double *part_buf, SolverScal *sc) {
  switch (part) {
    case 0: k64_ap<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, part_buf, sc); break;
    case 1: k64_s<<<cgrid(g), cblock(g), 0, s>>>(g, v, sc); break;
    case 2: k64_as<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, part_buf, sc); break;
    case 3: k64_xr<<<cgrid(g), cblock(g), 0, s>>>(g, v, part_buf, sc); break;
    default: k64_p<<<cgrid(g), cblock(g), 0, s>>>(g, v, sc); break;
  }
}

int loop64_blocks(long long ncell) {
  if (ncell > kLoopCells) return 0;
  // per device: 0 not asked yet, else blocks + 1 (a fact of the device and this build)
  constexpr int kDevices = 64;
  static std::atomic<int> known[kDevices];
  int dev = 0, nsm = 0, coop = 0, a = 0, b = 0, c = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
  if (const int k = known[dev].load()) return k - 1;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k64_bicg_loop<0>, kLoopBlock, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k64cg_loop, kLoopBlock, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k64_bicg_loop1, kLoopBlock, 0) != cudaSuccess)
    return 0;
  const int blocks = coop && a > 0 && b > 0 && c > 0 ? std::min(nsm, kLoopMaxBlocks) : 0;
  known[dev].store(blocks + 1);
  return blocks;
}
int loop64_iters(long long ncell) {
  const long long n = (1LL << 26) / (ncell > 0 ? ncell : 1);
  return (int)(n < 16 ? 16 : (n > 256 ? 256 : n));
}
size_t loop64_part_doubles() { return (size_t)kLoopSlots * kLoopMaxBlocks; }

// blocks, cells a block and shared memory of k32cg_loop; 0 blocks: not this grid (not uniform, too
// many cells for the multiprocessors' registers and shared memory) or device.  Every grid that fits
// takes it: against a kernel a phase, us an iteration, 28 grids of 37 K to 2.4 M cells measured 1.44
// to 2.35 times as fast, also where a plane is several times a block's range and each block forms p
// on both planes beside it: 8x150x160 (19 times) 9.8 / 14.7, 40x160x128 (3.8 times) 11.2 / 17.8; single
// cells, K = 16 (some registers spilled) 200x90x131 18.3 / 43.0, 16x110x110 (9.5 times) 11.5 / 16.7.
struct CgLoop {
  int blocks, chunk, v, k;
  size_t smem;
};
static CgLoop cg32_loop_plan(const Geo &g, const Stencil<float> &st, int nsm) {
  CgLoop P{};
  if (g.nonuni || st.jac || nsm < 1 || g.ncell > (long long)std::min(nsm, kLoopMaxBlocks) * kCgLoopBlock * kCgLoopCells)
    return P;
  for (int cls = 0; cls < 27; ++cls)  // one coefficient an axis side
    for (int e = 0; e < 7; ++e)
      if (e != 3 && st.c[cls][e] != 0.0f && st.c[cls][e] != st.c[13][e]) return P;
  const int sms = std::min(nsm, kLoopMaxBlocks);
  P.v = g.nzc % 4 == 0 ? 4 : 1;
  P.chunk = (int)(((g.ncell + sms - 1) / sms + 31) / 32 * 32);
  const int groups = (P.chunk / P.v + kCgLoopBlock - 1) / kCgLoopBlock;
  P.k = P.v == 4 ? (groups <= 1 ? 1 : groups <= 2 ? 2 : 4) : (groups <= 4 ? 4 : 16);
  P.smem = 4 * (2 * (size_t)g.nyc * g.nzc + 2 * (size_t)P.chunk);
  if (groups > P.k || P.smem > kCgLoopShared) return P;
  P.blocks = (int)((g.ncell + P.chunk - 1) / P.chunk);
  return P;
}
static void (*cg32_loop_kernel(const CgLoop &P))(Geo, Stencil<float>, Vec32, double *, SolverScal *, int, int) {
  if (P.v == 4) return P.k == 1 ? k32cg_loop<4, 1> : P.k == 2 ? k32cg_loop<4, 2> : k32cg_loop<4, 4>;
  return P.k == 4 ? k32cg_loop<1, 4> : k32cg_loop<1, 16>;
}
bool cg32_loop_fits(const Geo &g, const Stencil<float> &st, int nsm) {
  const CgLoop P = cg32_loop_plan(g, st, nsm);
  if (P.blocks == 0 || loop64_blocks(1) == 0) return false;  // (loop64_blocks: the device takes cooperative launches)
  int n = 0;
  const auto kernel = cg32_loop_kernel(P);
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCgLoopShared) == cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kCgLoopBlock, P.smem) == cudaSuccess && n >= 1;
}
void launch_cg32_loop(cudaStream_t s, const Geo &g, const Stencil<float> &st, KrylovVecs<float> v, float *const p2[2],
                      float *const ap2[2], double *part_buf, SolverScal *sc, int nsm) {
  const CgLoop P = cg32_loop_plan(g, st, nsm);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(P.blocks);
  cfg.blockDim = dim3(kCgLoopBlock);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, cg32_loop_kernel(P), g, st, v32(v, p2, ap2), part_buf, sc, kCg32LoopIters, P.chunk);
}

static void launch_loop(cudaStream_t s, bool cg, const Geo &g, const Stencil<double> &st, KrylovVecs<double> v,
                        double *part_buf, SolverScal *sc, int blocks, int iters) {
  // whole warps of cells a block, and no more blocks than hold any
  const long long chunk = ((g.ncell + blocks - 1) / blocks + 31) / 32 * 32;
  const int nb = (int)((g.ncell + chunk - 1) / chunk);
  const bool one = !cg && chunk <= kLoopBlock;  // a cell a thread
  auto kernel = cg        ? k64cg_loop
                : one     ? k64_bicg_loop1
                : !g.nonuni ? k64_bicg_loop<0>
                : st.jac  ? k64_bicg_loop<1>
                          : k64_bicg_loop<2>;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nb);
  cfg.blockDim = dim3(one ? (int)chunk : kLoopBlock);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, g, st, v, part_buf, sc, iters, (int)chunk);
}
void launch_bicg64_loop(cudaStream_t s, const Geo &g, const Stencil<double> &st, KrylovVecs<double> v,
                        double *part_buf, SolverScal *sc, int blocks, int iters) {
  launch_loop(s, false, g, st, v, part_buf, sc, blocks, iters);
}
void launch_cg64_loop(cudaStream_t s, const Geo &g, const Stencil<double> &st, KrylovVecs<double> v,
                      double *part_buf, SolverScal *sc, int blocks, int iters) {
  launch_loop(s, true, g, st, v, part_buf, sc, blocks, iters);
}

void launch_bicg32_part(cudaStream_t s, int part, const Geo &g, const Stencil<float> &st,
                        KrylovVecs<float> v, float *const p2[2], float *const ap2[2], double *part_buf,
                        SolverScal *sc) {
  const Vec32 w = v32(v, p2, ap2);
  if (g.tma && part < 2) {  // stencil kernels on the bulk-copy pipeline
    if (part == 0)
      k32t_pap<<<dim3(g.tgx, g.tgy, 1), kBlock, g.tsmem, s>>>(g, st, w, part_buf, sc);
    else
      k32t_sas<<<dim3(g.tgx, g.tgy2, 1), kBlock, g.tsmem2, s>>>(g, st, w, part_buf, sc);
    return;
  }
  if (g.vbx > 0) {  // vectorised path
    const dim3 vg(g.vgx, g.vgy, g.vgz), vb(g.vbx, g.vby, 1);
    switch (part) {
      case 0: k32v_pap<<<vg, vb, 0, s>>>(g, st, w, part_buf, sc); break;
      case 1: k32v_sas<<<vg, vb, 0, s>>>(g, st, w, part_buf, sc); break;
      default: k32v_xr<<<g.xgrid, kBlock, 0, s>>>(g, w, part_buf, sc); break;
    }
    return;
  }
  switch (part) {
    case 0: k32_pap<<<cgrid(g), cblock(g), 0, s>>>(g, st, w, part_buf, sc); break;
    case 1: k32_sas<<<cgrid(g), cblock(g), 0, s>>>(g, st, w, part_buf, sc); break;
    default: k32_xr<<<cgrid(g), cblock(g), 0, s>>>(g, w, part_buf, sc); break;
  }
}

void launch_bicgp32_part(cudaStream_t s, int part, const Geo &g, const Stencil<float> &st, PrecVecs v,
                         double *part_buf, SolverScal *sc) {
  if (g.vbx > 0) {  // quads
    const dim3 vg(g.vgx, g.vgy, g.vgz), vb(g.vbx, g.vby, 1);
    switch (part) {
      case 0: k32pv_p<<<g.xgrid, kBlock, 0, s>>>(g, v, sc); break;
      case 1: k32pv_v<<<vg, vb, 0, s>>>(g, st, v, part_buf, sc); break;
      case 2: k32pv_s<<<g.xgrid, kBlock, 0, s>>>(g, v, sc); break;
      case 3: k32pv_t<<<vg, vb, 0, s>>>(g, st, v, part_buf, sc); break;
      default: k32pv_xr<<<g.xgrid, kBlock, 0, s>>>(g, v, part_buf, sc); break;
    }
    return;
  }
  switch (part) {
    case 0: k32p_p<<<cgrid(g), cblock(g), 0, s>>>(g, v, sc); break;
    case 1: k32p_v<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, part_buf, sc); break;
    case 2: k32p_s<<<cgrid(g), cblock(g), 0, s>>>(g, v, sc); break;
    case 3: k32p_t<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, part_buf, sc); break;
    default: k32p_xr<<<cgrid(g), cblock(g), 0, s>>>(g, v, part_buf, sc); break;
  }
}

void launch_cg_setup64(cudaStream_t s, const Geo &g, const Stencil<double> &st, KrylovVecs<double> v, const double *b,
                       double *px1, double *px2, double *part, SolverScal *sc) {
  k64cg_setup<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, b, px1, px2, part, sc);
}
void launch_cg64_part(cudaStream_t s, int part, const Geo &g, const Stencil<double> &st, KrylovVecs<double> v,
                      double *part_buf, SolverScal *sc) {
  switch (part) {
    case 0: k64cg_q<<<cgrid(g), cblock(g), 0, s>>>(g, st, v, part_buf, sc); break;
    case 1: k64cg_xr<<<cgrid(g), cblock(g), 0, s>>>(g, v, part_buf, sc); break;
    default: k64cg_p<<<cgrid(g), cblock(g), 0, s>>>(g, v, sc); break;
  }
}
void launch_cg32_part(cudaStream_t s, int part, const Geo &g, const Stencil<float> &st, KrylovVecs<float> v,
                      float *const p2[2], float *const ap2[2], double *part_buf, SolverScal *sc) {
  const Vec32 w = v32(v, p2, ap2);
  if (part == 1) {
    const int grid = g.xgrid > 0 ? g.xgrid : g.lgx * g.lgy * g.lgz;
    k32cg_xr<<<grid, kBlock, 0, s>>>(g, w, part_buf, sc);
  } else if (g.tma) {
    k32cgt_pq<<<dim3(g.tgx, g.tgy2, 1), kBlock, g.tsmem2, s>>>(g, st, w, part_buf, sc);
  } else if (g.vbx > 0) {
    k32cgv_pq<<<dim3(g.vgx, g.vgy, g.vgz), dim3(g.vbx, g.vby, 1), 0, s>>>(g, st, w, part_buf, sc);
  } else {
    k32cg_pq<<<cgrid(g), cblock(g), 0, s>>>(g, st, w, part_buf, sc);
  }
}
void launch_bicg_nan_reset(cudaStream_t s, int, const Geo &g, double *x, const double *px1, const double *px2,
                           double *part, SolverScal *sc) {
  k_nan_replace<<<cgrid(g), cblock(g), 0, s>>>(g, x, px1, part, sc);
  k_nan_restore<<<cgrid(g), cblock(g), 0, s>>>(g, x, px2, sc);
}

// the integer form covers the grid: pairs along k, a plane's and two rows' offsets in 32 bits,
// spacings its exponents are safe with, and none so much wider than another that its weight, in
// units of the largest one's, keeps fewer than FP64's 53 bits (cells of about 11 : 1)
static long long fix_weight(double w, int k) { return std::llround(std::ldexp(w, k)); }
static int fix_exponent(const double (&w)[3]) { return 59 - std::ilogb(std::max(w[0], std::max(w[1], w[2]))); }
static bool fix_residual(const Geo &g) {
  if (g.nonuni || g.nzc % 2 != 0 || g.nzc < 4 || (long long)g.nyc * g.nzc >= (1LL << 30)) return false;
  for (double h : {g.hx, g.hy, g.hz})
    if (!(h > 1e-9 && h < 1e9)) return false;
  const double w[3] = {1.0 / (g.hx * g.hx), 1.0 / (g.hy * g.hy), 1.0 / (g.hz * g.hz)};
  return fix_weight(std::min(w[0], std::min(w[1], w[2])), fix_exponent(w)) >= 1LL << 52;
}
// the integer form's operator: w_a times the power of two that brings the largest below 2^60
static FixOp fix_op(const Geo &g, const Stencil<float> &st32) {
  FixOp F{};
  const double w[3] = {1.0 / (g.hx * g.hx), 1.0 / (g.hy * g.hy), 1.0 / (g.hz * g.hz)};
  F.k = fix_exponent(w);
  for (int a = 0; a < 3; ++a) {
    const long long q = fix_weight(w[a], F.k);
    F.wh[a] = (unsigned)(q >> 30);
    F.wl[a] = (unsigned)(q & 0x3fffffff);
  }
  for (int q = 0; q < 27; ++q) F.dg[q] = st32.dg[q];
  return F;
}
void launch_residual64(cudaStream_t s, int nsm, const Geo &g, const Stencil<double> &st, const Stencil<float> &st32,
                       int jacobi, const double *b, const double *x, float *rf, double *part, StepScal *ss,
                       SolverScal *inner, int flags, bool chain) {
  if (!chain && fix_residual(g)) {
    const FixOp F = fix_op(g, st32);
    int bx = 1;
    while (bx < g.nzc / 2 && bx < 32) bx *= 2;
    const dim3 block(bx, kBlock / bx);
    dim3 grid((g.nzc / 2 + bx - 1) / bx, ((g.nyc + 1) / 2 + block.y - 1) / block.y, 1);
    // segments of planes for whole waves of two blocks a multiprocessor, each with a plane before it
    const int tiles = (int)(grid.x * grid.y), wave = 2 * nsm;
    long long best = 0;
    for (int w = 1; w <= 6; ++w) {
      const int z = std::max(1, std::min(g.nxc, w * wave / tiles)), chunk = (g.nxc + z - 1) / z;
      const int nz = (g.nxc + chunk - 1) / chunk;
      const long long cost = (long long)((tiles * (long long)nz + wave - 1) / wave) * (chunk + 1);
      if (best && cost >= best) continue;
      best = cost;
      grid.z = nz;
    }
    (flags & 1 ? k_residual_fx<true> : k_residual_fx<false>)<<<grid, block, 0, s>>>(g, st, F, jacobi, b, x, rf, part, ss,
                                                                                    inner, flags);
    return;
  }
  if (flags & 1)
    k_residual64<true><<<cgrid(g), cblock(g), 0, s>>>(g, st, jacobi, b, x, rf, part, ss, inner, flags);
  else
    k_residual64<false><<<cgrid(g), cblock(g), 0, s>>>(g, st, jacobi, b, x, rf, part, ss, inner, flags);
}
void launch_refine_start32(cudaStream_t s, const Geo &g, const Stencil<double> &st, int jacobi, KrylovVecs<float> v,
                           float *const p2[2], float *const ap2[2], const float *rf, const StepScal *ss,
                           double delta, double peak, int first, double *part, SolverScal *sc) {
  k_refine_start32<<<cgrid(g), cblock(g), 0, s>>>(g, st, jacobi, v32(v, p2, ap2), rf, ss, delta, peak, first, part,
                                                   sc);
}
void launch_sum32(cudaStream_t s, const Geo &g, const float *e, double *part, StepScal *ss) {
  k_sum32<<<g.xgrid, kBlock, 0, s>>>(g, e, part, ss);
}
void launch_correct64(cudaStream_t s, int, const Geo &g, double *x, const float *e, double factor,
                      const StepScal *ss) {
  // factor = +-2^k (sweep_scale); a zero factor (a zero residual, never corrected) adds nothing
  if (!(std::fabs(factor) > 0.0) || !std::isfinite(factor)) return;
  k_correct64<<<g.xgrid, kBlock, 0, s>>>(g, x, e, std::ilogb(factor), factor < 0.0 ? 1 : 0, ss);
}
void launch_project_rhs(cudaStream_t s, const Geo &g, const Stencil<double> &st, int jacobi, double *b, double *part,
                        StepScal *ss) {
  k_rhs_sum<<<cgrid(g), cblock(g), 0, s>>>(g, st, jacobi, b, part, ss);
  k_rhs_subtract<<<cgrid(g), cblock(g), 0, s>>>(g, st, jacobi, b, ss);
}
void launch_scale_rows(cudaStream_t s, const Geo &g, const Stencil<double> &st, int jacobi, const double *in,
                       double *out) {
  k_scale_rows<<<cgrid(g), cblock(g), 0, s>>>(g, st, jacobi, in, out);
}
void launch_rbsor_sweep(cudaStream_t s, int, const Geo &g, const Stencil<double> &st, const double *b, double *x,
                        double omega) {
  k_rbsor<<<cgrid(g), cblock(g), 0, s>>>(g, st, b, x, omega, 0);
  k_rbsor<<<cgrid(g), cblock(g), 0, s>>>(g, st, b, x, omega, 1);
}
void launch_residual_norm64(cudaStream_t s, int, const Geo &g, const Stencil<double> &st, const double *b,
                            const double *x, double *part, StepScal *ss) {
  k_residual_norm64<<<cgrid(g), cblock(g), 0, s>>>(g, st, b, x, part, ss);
}
void launch_vec_norm64(cudaStream_t s, int, const Geo &g, const double *b, double *part, StepScal *ss) {
  k_vec_norm64<<<cgrid(g), cblock(g), 0, s>>>(g, b, part, ss);
}

}  // namespace cfdgb
