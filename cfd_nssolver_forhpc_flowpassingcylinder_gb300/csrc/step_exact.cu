// FP64 projection-step kernels that reproduce the reference's arithmetic exactly.
//
// This translation unit is compiled with -fmad=false and IEEE division, so every
// kernel performs the reference function's operations in the same order and rounding:
// the results are bit-identical to the reference (checked against its golden vectors).
// One thread per interior cell (grid-stride over compact rows, k fastest, so a warp
// reads contiguous k runs of each padded array).
#include <algorithm>
#include <cmath>

#include "cfdgb_internal.cuh"
#include "reduce.cuh"
#include "stepctl.cuh"
#include "kernels.h"

namespace cfdgb {

// inc/source/Convection_Difussion.hpp:96-147 (LudUnitA; LudUnitB has the same body)
__device__ __forceinline__ void lud(bool two, double Up, double Un, long long pp, long long p, long long ic, long long n,
                                    long long nn, const double *__restrict__ Di, const double *__restrict__ Ds,
                                    const double *__restrict__ rDi, const double *__restrict__ rDs, int I,
                                    const double *__restrict__ phi, double &P, double &N) {
  const double fc = phi[ic], fp = phi[p], fn = phi[n];
  auto oi = [&](double a, int q) { return div_by(a, Di[q], rDi[q], two); };  // a / Di[q]
  if (Up > 0.0)
    P = (fc + oi(0.5 * Ds[I] * (fc - fn), I));
  else
    P = (fp + oi(0.5 * Ds[I + 1] * (fp - phi[pp]), I + 1));
  if (Un > 0.0)
    N = (fn + oi(0.5 * Ds[I - 1] * (fn - phi[nn]), I - 1));
  else
    N = (fc + oi(0.5 * Ds[I] * (fc - fp), I + 1));
}

// face values of one axis under the convection switch (inc/0_General.hpp:114-118): LUD or UD
// (UdUnit, :150-168; QUICK is k_convdiff_quick)
template <int S>
__device__ __forceinline__ void face(bool two, double Up, double Un, long long pp, long long p, long long ic, long long n,
                                     long long nn, const double *__restrict__ Di, const double *__restrict__ Ds,
                                     const double *__restrict__ rDi, const double *__restrict__ rDs, int I,
                                     const double *__restrict__ phi, double &P, double &N) {
  if (S == CFDGB_LUD) {
    lud(two, Up, Un, pp, p, ic, n, nn, Di, Ds, rDi, rDs, I, phi, P, N);
  } else {
    P = Up > 0.0 ? phi[ic] : phi[p];
    N = Un > 0.0 ? phi[n] : phi[ic];
  }
}

// inc/source/SmagorinskyModel.hpp:30-79 with GradientGauss (:6-26), CS = 0.18: eddy
// viscosity of T0 per cell, nut[row] = l2[row] sqrt|2 ux^2 + vy^2 + wz^2 + (uy + vx)^2 +
// (uz + wx)^2 + (vz + wy)^2| with the reference's central differences (u over Dxs, Dy, Dz;
// v over Dx, Dys, Dz; w over Dx, Dy, Dzs; the sum as the reference writes it).  l2 =
// (CS cbrt(Dx Dy Dz))^2 per cell, computed once on the host with the same pow.
__global__ void __launch_bounds__(kBlock) k_smagorinsky(Geo g, const double *__restrict__ l2,
                                                        const double *__restrict__ u, const double *__restrict__ v,
                                                        const double *__restrict__ w, double *__restrict__ nut) {
  const long long sx = g.sx, sy = g.sy;
  for (long long row = blockIdx.x * (long long)kBlock + threadIdx.x; row < g.ncell;
       row += (long long)gridDim.x * kBlock) {
    int i, j, k;
    row_ijk(g, row, i, j, k);
    const long long c = pidx(g, i, j, k);
    const bool two = g.div2 != 0;
    auto h = [&](double d, double r) { return div_by(0.5, d, r, two); };  // 0.5 / d
    const double ux = h(g.Dxs[i], g.rDxs[i]) * (u[c - sx] - u[c + sx]);
    const double uy = h(g.Dy[j], g.rDy[j]) * (u[c - sy] - u[c + sy]);
    const double uz = h(g.Dz[k], g.rDz[k]) * (u[c - 1] - u[c + 1]);
    const double vx = h(g.Dx[i], g.rDx[i]) * (v[c - sx] - v[c + sx]);
    const double vy = h(g.Dys[j], g.rDys[j]) * (v[c - sy] - v[c + sy]);
    const double vz = h(g.Dz[k], g.rDz[k]) * (v[c - 1] - v[c + 1]);
    const double wx = h(g.Dx[i], g.rDx[i]) * (w[c - sx] - w[c + sx]);
    const double wy = h(g.Dy[j], g.rDy[j]) * (w[c - sy] - w[c + sy]);
    const double wz = h(g.Dzs[k], g.rDzs[k]) * (w[c - 1] - w[c + 1]);
    const double a = uy + vx, b = uz + wx, e = vz + wy;
    const double temp = fabs(2.0 * (ux * ux) + vy * vy + wz * wz + a * a + b * b + e * e);
    nut[row] = l2[row] * sqrt(temp);
  }
}

// inc/source/Convection_Difussion.hpp:174-450: explicit Euler convection (LUD or UD here)
// + central diffusion; the last face along a component's own axis is a boundary face and
// skipped.
// S: the convection scheme; nut (compact, may be null): the Smagorinsky eddy viscosity
// added to nu per cell (Convection_Difussion.hpp:251-256).
// Fused with get_Cfl (inc/analyses/cfl.hpp:3-78, called on u* right after this function,
// src/RUN_CPU.cpp:274): each thread takes u*, v*, w* of its cell from registers, with the
// reference's division and order (c = u/Dxs + v/Dys + w/Dzs, a term left out on the last
// face of its axis), so the CFL number and extremes are those of get_Cfl bit for bit; the
// maxima are exact in any order.  The last block also sets the next dt (StepCtl).
// Two resident blocks per SM (at most 128 registers a thread): the kernel is bound by the
// FP64 pipe, and one block of 8 warps per SM leaves it waiting on latency.
template <int S, bool AB>
__global__ void __launch_bounds__(kBlock, 2) k_convdiff_exact(Geo g, double dt_arg, double nu0,
                                                           const double *__restrict__ nut,
                                                           const double *__restrict__ u,
                                                           const double *__restrict__ v,
                                                           const double *__restrict__ w,
                                                           double *__restrict__ us,
                                                           double *__restrict__ vs,
                                                           double *__restrict__ ws, StepCtl sc) {
  const double dt = step_dt(sc, dt_arg);
  const bool two = g.div2 != 0;
  CflAcc cfl;
  AbStep ab;
  if (AB) ab.init(sc, dt);
  const long long sx = g.sx, sy = g.sy, sz = 1;
  const double *Dx = g.Dx, *Dy = g.Dy, *Dz = g.Dz, *Dxs = g.Dxs, *Dys = g.Dys, *Dzs = g.Dzs;
  const double *rDx = g.rDx, *rDy = g.rDy, *rDz = g.rDz, *rDxs = g.rDxs, *rDys = g.rDys, *rDzs = g.rDzs;
  // a / D[q] of each metric array (div_by with the array's reciprocals)
  auto ox = [&](double a, int q) { return div_by(a, Dx[q], rDx[q], two); };
  auto oy = [&](double a, int q) { return div_by(a, Dy[q], rDy[q], two); };
  auto oz = [&](double a, int q) { return div_by(a, Dz[q], rDz[q], two); };
  auto oxs = [&](double a, int q) { return div_by(a, Dxs[q], rDxs[q], two); };
  auto oys = [&](double a, int q) { return div_by(a, Dys[q], rDys[q], two); };
  auto ozs = [&](double a, int q) { return div_by(a, Dzs[q], rDzs[q], two); };
  for (long long row = blockIdx.x * (long long)kBlock + threadIdx.x; row < g.ncell;
       row += (long long)gridDim.x * kBlock) {
    int i, j, k;
    row_ijk(g, row, i, j, k);
    const long long ic = pidx(g, i, j, k);
    const double nu = nut ? nu0 + nut[row] : nu0;
    const long long xm = ic - sx, xp = ic + sx, ym = ic - sy, yp = ic + sy, zm = ic - sz, zp = ic + sz;
    double ccfl = 0.0;
    if (i < g.nx - 3) {  // u
      const double IT = ox(Dxs[i] * 0.5, i);
      const double uc = u[ic], uxp = u[xp], uxm = u[xm];
      const double Up = 0.5 * (uxp + uc);
      const double Un = 0.5 * (uxm + uc);
      const double Vp = v[ic] + (v[xp] - v[ic]) * IT;
      const double Vn = v[ym] + (v[ym + xp - ic] - v[ym]) * IT;
      const double Wp = w[ic] + (w[xp] - w[ic]) * IT;
      const double Wn = w[zm] + (w[zm + xp - ic] - w[zm]) * IT;
      double uPx, uNx, uPy, uNy, uPz, uNz;
      face<S>(two, Up, Un, ic + 2 * sx, xp, ic, xm, ic - 2 * sx, Dx, Dxs, rDx, rDxs, i, u, uPx, uNx);
      face<S>(two, Vp, Vn, ic + 2 * sy, yp, ic, ym, ic - 2 * sy, Dy, Dys, rDy, rDys, j, u, uPy, uNy);
      face<S>(two, Wp, Wn, ic + 2 * sz, zp, ic, zm, ic - 2 * sz, Dz, Dzs, rDz, rDzs, k, u, uPz, uNz);
      const double convection = -dt * (oxs(uPx * uPx - uNx * uNx, i) + oy(uPy * Vp - uNy * Vn, j) +
                                       oz(uPz * Wp - uNz * Wn, k));
      const double difussion =
          nu * dt *
          (oxs(ox(uxp - uc, i + 1) - ox(uc - uxm, i), i) +
           oy(oys(u[yp] - uc, j) - oys(uc - u[ym], j - 1), j) +
           oz(ozs(u[zp] - uc, k) - ozs(uc - u[zm], k - 1), k));
      const double r = AB ? ab.value(0, ic, uc, convection, difussion) : uc + convection + difussion;
      us[ic] = r;
      ccfl += oxs(r, i);
      cfl.comp(0, r);
    }
    if (j < g.ny - 3) {  // v
      const double IT = oy(Dys[j] * 0.5, j);
      const double vc = v[ic], vyp = v[yp], vym = v[ym];
      const double Vp = 0.5 * (vyp + vc);
      const double Vn = 0.5 * (vym + vc);
      const double Up = u[ic] + (u[yp] - u[ic]) * IT;
      const double Un = u[xm] + (u[xm + yp - ic] - u[xm]) * IT;
      const double Wp = w[ic] + (w[yp] - w[ic]) * IT;
      const double Wn = w[zm] + (w[zm + yp - ic] - w[zm]) * IT;
      double vPx, vNx, vPy, vNy, vPz, vNz;
      face<S>(two, Up, Un, ic + 2 * sx, xp, ic, xm, ic - 2 * sx, Dx, Dxs, rDx, rDxs, i, v, vPx, vNx);
      face<S>(two, Vp, Vn, ic + 2 * sy, yp, ic, ym, ic - 2 * sy, Dy, Dys, rDy, rDys, j, v, vPy, vNy);
      face<S>(two, Wp, Wn, ic + 2 * sz, zp, ic, zm, ic - 2 * sz, Dz, Dzs, rDz, rDzs, k, v, vPz, vNz);
      const double convection = -dt * (ox(Up * vPx - Un * vNx, i) + oys(vPy * vPy - vNy * vNy, j) +
                                       oz(Wp * vPz - Wn * vNz, k));
      const double difussion =
          nu * dt *
          (ox(oxs(v[xp] - vc, i) - oxs(vc - v[xm], i - 1), i) +
           oys(oy(vyp - vc, j + 1) - oy(vc - vym, j), j) +
           oz(ozs(v[zp] - vc, k) - ozs(vc - v[zm], k - 1), k));
      const double r = AB ? ab.value(1, ic, vc, convection, difussion) : vc + convection + difussion;
      vs[ic] = r;
      ccfl += oys(r, j);
      cfl.comp(1, r);
    }
    if (k < g.nz - 3 + g.pz) {  // w (periodic z: the top face too)
      const double IT = oz(Dzs[k] * 0.5, k);
      const double wc = w[ic], wzp = w[zp], wzm = w[zm];
      const double Wp = 0.5 * (wzp + wc);
      const double Wn = 0.5 * (wzm + wc);
      const double Up = u[ic] + (u[zp] - u[ic]) * IT;
      const double Un = u[xm] + (u[xm + zp - ic] - u[xm]) * IT;
      const double Vp = v[ic] + (v[zp] - v[ic]) * IT;
      const double Vn = v[ym] + (v[ym + zp - ic] - v[ym]) * IT;
      double wPx, wNx, wPy, wNy, wPz, wNz;
      face<S>(two, Up, Un, ic + 2 * sx, xp, ic, xm, ic - 2 * sx, Dx, Dxs, rDx, rDxs, i, w, wPx, wNx);
      face<S>(two, Vp, Vn, ic + 2 * sy, yp, ic, ym, ic - 2 * sy, Dy, Dys, rDy, rDys, j, w, wPy, wNy);
      face<S>(two, Wp, Wn, ic + 2 * sz, zp, ic, zm, ic - 2 * sz, Dz, Dzs, rDz, rDzs, k, w, wPz, wNz);
      const double convection = -dt * (ox(Up * wPx - Un * wNx, i) + oy(Vp * wPy - Vn * wNy, j) +
                                       ozs(wPz * wPz - wNz * wNz, k));
      const double difussion =
          nu * dt *
          (ox(oxs(w[xp] - wc, i) - oxs(wc - w[xm], i - 1), i) +
           oy(oys(w[yp] - wc, j) - oys(wc - w[ym], j - 1), j) +
           ozs(oz(wzp - wc, k + 1) - oz(wc - wzm, k), k));
      const double r = AB ? ab.value(2, ic, wc, convection, difussion) : wc + convection + difussion;
      ws[ic] = r;
      ccfl += ozs(r, k);
      cfl.comp(2, r);
    }
    cfl.cell(ccfl);
  }
  if (sc.ss) cfl_finish(cfl, dt, sc);
}

// The same for QUICK (QuickUnitA and QuickUnitB, Convection_Difussion.hpp:20-90), with every face
// computed once.  The kernel is bound by the FP64 pipe (one warp instruction per 64 cycles and
// scheduler, idle lanes included), so what counts is the number of FP64 instructions a cell: in the
// per-cell form above both faces of each axis (every face twice), up to four divisions of
// every difference and the QUICK factors' divisions took about 1050; here
//   - a block of (tk + 2) x (rows + 1) threads marches along x, a thread owning one (j, k)
//     column: the x face of plane i is kept in registers as the lower face of plane i + 1;
//   - the differences and the upper faces along y and z go through shared memory to the
//     neighbouring threads (two buffers each, one barrier a plane: the next plane's
//     differences are formed before the barrier that publishes this plane's faces).  The first
//     row and the first lane of a row hold no cell and compute the faces below the tile, the
//     last lane the difference above it;
//   - the factors 0.125 D^2 / Ds come from tables (Geo::qk*, each IEEE division's result);
// about 215 instructions a cell.  Every value is formed by the reference's operations in its
// order, so the results are the same bits (a face's value, velocity and flux are the same
// expression from both of its cells).  512x256x64: 16.6 -> 4.9 ms (85 % of the FP64 pipe).
struct QuickPlan {
  int tk, rows, xc;      // cells of a tile along k and j, planes a block marches over
  int threads, gx, gy, gz;
};

// The upper QUICK face's flux on one axis: the value fc and the next one fp, the differences
// s0 = d0 - dm around the value and s1 around the next one, the factors of the two flow
// directions and the face velocity vel (own axis: the face's own mean).
template <bool OWN>
__device__ __forceinline__ double quick_flux(double mean, double s0, double s1, double kp, double kn, double vel) {
  const bool up = positive(vel);
  const double P = mean - (up ? kp : kn) * (up ? s0 : s1);
  return OWN ? P * P : P * vel;
}

template <bool AB, bool TWO>
__global__ void __launch_bounds__(512, 1) k_convdiff_quick(Geo g, QuickPlan pl, double dt_arg, double nu0,
                                                           const double *__restrict__ nut,
                                                           const double *__restrict__ u,
                                                           const double *__restrict__ v,
                                                           const double *__restrict__ w, double *__restrict__ us,
                                                           double *__restrict__ vs, double *__restrict__ ws,
                                                           StepCtl sc) {
  extern __shared__ double qsm[];
  const int T = blockDim.x, t = threadIdx.x, W = pl.tk + 2;
  double *sd = qsm + t, *sf = qsm + 12 * T + t;  // differences and fluxes: [buffer][y, z of u, v, w][thread]
  const double dt = step_dt(sc, dt_arg);
  CflAcc cfl;
  AbStep ab;
  if (AB) ab.init(sc, dt);
  const int tr = t / W, tc = t - tr * W;
  const int j = 1 + blockIdx.y * pl.rows + tr, k = 1 + blockIdx.x * pl.tk + tc;
  const bool row = tr <= pl.rows && j <= g.ny - 3;
  const bool in = row && tc <= pl.tk && k <= g.nz - 3;
  const bool yf = in && tc > 0, zf = in && tr > 0, cell = yf && zf;
  const bool zd = row && tr > 0 && k <= g.nz - 2;  // the difference to the next cell along k
  const bool jtop = tr == pl.rows || j == g.ny - 3;  // no thread above holds the next difference
  const int sx = (int)g.sx, sy = (int)g.sy;  // offsets within a plane or two: below 2^31 entries
  const int i0 = 2 + blockIdx.z * pl.xc, i1 = min(g.nx - 2, i0 + pl.xc);
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const double *qx = g.qkx, *qy = g.qky, *qz = g.qkz;  // rows: own axis up, down; across up, down
  const int jj = row ? j : 2, kk = in || zd ? k : 2;
  long long c = (long long)i0 * g.sx + (long long)jj * sy + kk;
  const double hy = g.hfy[jj], hz = g.hfz[kk];
  const double nudt0 = nu0 * dt;
  auto over = [](double a, const double *D, const double *rD, int q) { return div_by(a, D[q], rD[q], TWO); };
  const double *const ph[3] = {u, v, w};
  // the spacings that divide a difference (to the next value) along an axis, own or across
  const double *const Sx[3] = {g.Dx + 1, g.Dxs, g.Dxs}, *const rSx[3] = {g.rDx + 1, g.rDxs, g.rDxs};
  const double *const Sy[3] = {g.Dys, g.Dy + 1, g.Dys}, *const rSy[3] = {g.rDys, g.rDy + 1, g.rDys};
  const double *const Sz[3] = {g.Dzs, g.Dzs, g.Dz + 1}, *const rSz[3] = {g.rDzs, g.rDzs, g.rDz + 1};
  // differences of plane cc along y and z, into buffer s
  auto differences = [&](const double (&f)[3], long long cc, double *s) {
    if (yf) {
#pragma unroll
      for (int a = 0; a < 3; ++a) s[a * T] = over(ph[a][cc + sy] - f[a], Sy[a], rSy[a], j);
    }
    if (zd) {
#pragma unroll
      for (int a = 0; a < 3; ++a) s[(3 + a) * T] = over(ph[a][cc + 1] - f[a], Sz[a], rSz[a], k);
    }
  };
  // x faces: the value, the difference and the flux of the plane before, per component
  double fu[3] = {0, 0, 0}, dx[3] = {0, 0, 0}, fx[3] = {0, 0, 0};
  if (in || zd) {
#pragma unroll
    for (int a = 0; a < 3; ++a) fu[a] = ph[a][c];
  }
  if (cell) {  // the face below the first plane
    const long long m = c - sx;
    const int i = i0 - 1;
    const double um = u[m];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double *f = ph[a] + m;
      const double f0 = f[0], d0 = over(fu[a] - f0, Sx[a], rSx[a], i);
      const double s0 = d0 - over(f0 - f[-sx], Sx[a], rSx[a], i - 1);
      const double s1 = over(f[2 * sx] - fu[a], Sx[a], rSx[a], i + 1) - d0;
      const double mean = 0.5 * (f0 + fu[a]), vel = a == 1 ? um + (u[m + sy] - um) * hy : um + (u[m + 1] - um) * hz;
      fx[a] = a == 0 ? quick_flux<true>(mean, s0, s1, qx[i], qx[nx + i], mean)
                     : quick_flux<false>(mean, s0, s1, qx[2 * nx + i], qx[3 * nx + i], vel);
      dx[a] = d0;
    }
  }
  differences(fu, c, sd);
  __syncthreads();
  for (int i = i0; i < i1; ++i, c += sx) {
    double fn[3] = {0, 0, 0}, sy0[3], sz0[3];  // next plane's values; second differences along y and z
    if (in || zd) {
#pragma unroll
      for (int a = 0; a < 3; ++a) fn[a] = ph[a][c + sx];
    }
    const double hx = g.hfx[i];
    if (yf) {
      const double vx = fu[1] + (fn[1] - fu[1]) * hx, vz = fu[1] + (v[c + 1] - fu[1]) * hz;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double fp = ph[a][c + sy], d0 = sd[a * T];
        const double dm = tr > 0 ? sd[a * T - W] : over(fu[a] - ph[a][c - sy], Sy[a], rSy[a], j - 1);
        const double dp = !jtop ? sd[a * T + W] : over(ph[a][c + 2 * sy] - fp, Sy[a], rSy[a], j + 1);
        const double mean = 0.5 * (fu[a] + fp);
        sy0[a] = d0 - dm;
        sf[a * T] = a == 1 ? quick_flux<true>(mean, sy0[a], dp - d0, qy[j], qy[ny + j], mean)
                           : quick_flux<false>(mean, sy0[a], dp - d0, qy[2 * ny + j], qy[3 * ny + j], a == 0 ? vx : vz);
      }
    }
    if (zf) {
      const double wx = fu[2] + (fn[2] - fu[2]) * hx, wy = fu[2] + (w[c + sy] - fu[2]) * hy;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double fp = ph[a][c + 1], d0 = sd[(3 + a) * T], dp = sd[(3 + a) * T + 1];
        const double dm = tc > 0 ? sd[(3 + a) * T - 1] : over(fu[a] - ph[a][c - 1], Sz[a], rSz[a], k - 1);
        const double mean = 0.5 * (fu[a] + fp);
        sz0[a] = d0 - dm;
        sf[(3 + a) * T] =
            a == 2 ? quick_flux<true>(mean, sz0[a], dp - d0, qz[k], qz[nz + k], mean)
                   : quick_flux<false>(mean, sz0[a], dp - d0, qz[2 * nz + k], qz[3 * nz + k], a == 0 ? wx : wy);
      }
    }
    double *const so = qsm + t + (((i - i0) & 1) ? 0 : 6 * T);  // the other buffer of differences
    if (i + 1 < i1) differences(fn, c + sx, so);
    __syncthreads();
    if (cell) {
      double nudt = nudt0;
      if (nut) nudt = (nu0 + nut[((long long)(i - 2) * g.nyc + (j - 2)) * g.nzc + (k - 2)]) * dt;
      double ccfl = 0.0;
      const double uy = fu[0] + (u[c + sy] - fu[0]) * hy, uz = fu[0] + (u[c + 1] - fu[0]) * hz;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        // the x face; its third difference only in warps with flow from that side
        const double d0 = over(fn[a] - fu[a], Sx[a], rSx[a], i), s0 = d0 - dx[a];
        const double mean = 0.5 * (fu[a] + fn[a]), vel = a == 0 ? mean : a == 1 ? uy : uz;
        double s1 = s0;
        if (__any_sync(__activemask(), !positive(vel)))
          s1 = over(ph[a][c + 2 * sx] - fn[a], Sx[a], rSx[a], i + 1) - d0;
        const double F = a == 0 ? quick_flux<true>(mean, s0, s1, qx[i], qx[nx + i], vel)
                                : quick_flux<false>(mean, s0, s1, qx[2 * nx + i], qx[3 * nx + i], vel);
        const bool on = a == 0 ? i < nx - 3 : a == 1 ? j < ny - 3 : k < nz - 3 + g.pz;
        if (on) {
          // the spacings between the component's own faces, per axis
          const double *ax = a == 0 ? g.Dxs : g.Dx, *rax = a == 0 ? g.rDxs : g.rDx;
          const double *ay = a == 1 ? g.Dys : g.Dy, *ray = a == 1 ? g.rDys : g.rDy;
          const double *az = a == 2 ? g.Dzs : g.Dz, *raz = a == 2 ? g.rDzs : g.rDz;
          const double convection = -dt * (over(F - fx[a], ax, rax, i) + over(sf[a * T] - sf[a * T - W], ay, ray, j) +
                                           over(sf[(3 + a) * T] - sf[(3 + a) * T - 1], az, raz, k));
          const double difussion =
              nudt * (over(s0, ax, rax, i) + over(sy0[a], ay, ray, j) + over(sz0[a], az, raz, k));
          const double r = AB ? ab.value(a, c, fu[a], convection, difussion) : fu[a] + convection + difussion;
          (a == 0 ? us : a == 1 ? vs : ws)[c] = r;
          ccfl += a == 0 ? over(r, g.Dxs, g.rDxs, i) : a == 1 ? over(r, g.Dys, g.rDys, j) : over(r, g.Dzs, g.rDzs, k);
          cfl.comp(a, r);
        }
        dx[a] = d0;
        fx[a] = F;
      }
      cfl.cell(ccfl);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) fu[a] = fn[a];
    sd = so;
    sf = qsm + 12 * T + t + (((i - i0) & 1) ? 0 : 6 * T);
  }
  if (sc.ss) cfl_finish(cfl, dt, sc);
}

// Tiles of k_convdiff_quick: whole k lines up to 126 cells, as many rows as 512 threads hold,
// and the number of x chunks (one plane's face of extra work each) that costs least in whole
// waves of one block a multiprocessor.
static QuickPlan quick_plan(const Geo &g, int nsm) {
  QuickPlan p;
  const int kt = (g.nzc + 125) / 126;
  p.tk = (g.nzc + kt - 1) / kt;
  const int rows = std::min(g.nyc, 512 / (p.tk + 2) - 1);
  p.gy = (g.nyc + rows - 1) / rows;
  p.rows = (g.nyc + p.gy - 1) / p.gy;
  p.gx = (g.nzc + p.tk - 1) / p.tk;
  p.threads = ((p.tk + 2) * (p.rows + 1) + 31) / 32 * 32;
  double best = 1e300;
  p.xc = g.nxc;
  const int most = std::min(g.nxc, std::max(1, kConvdiffBlocks * nsm / (p.gx * p.gy)));
  for (int n = 1; n <= most; ++n) {
    const int xc = (g.nxc + n - 1) / n, nb = (g.nxc + xc - 1) / xc;
    const double cost = std::ceil((double)nb * p.gx * p.gy / nsm) * (xc + 0.4);
    if (cost < best) {
      best = cost;
      p.xc = xc;
    }
  }
  p.gz = (g.nxc + p.xc - 1) / p.xc;
  return p;
}

// inc/matrix/b_matrix.hpp:35-98: b = -(jp)(1/dt) div(u*), one-sided differences
// TWO: div_by's double correction (a template, as the branch would be predicated: two more FP64
// instructions a division)
template <bool TWO>
__global__ void __launch_bounds__(kBlock) k_rhs_exact(Geo g, double dt_arg, const double *dtp,
                                                      const double *__restrict__ us,
                                                      const double *__restrict__ vs,
                                                      const double *__restrict__ ws, int jacobi,
                                                      Stencil<double> st, double *__restrict__ b) {
  const double ddt = 1.0 / (dtp ? *dtp : dt_arg);
  for (long long row = blockIdx.x * (long long)kBlock + threadIdx.x; row < g.ncell;
       row += (long long)gridDim.x * kBlock) {
    int i, j, k;
    row_ijk(g, row, i, j, k);
    const long long ic = pidx(g, i, j, k);
    // periodic z: the bottom face of the first cell is the top face nz-3
    const long long zb = (g.pz && k == 2) ? ic + g.nzc - 1 : ic - 1;
    const double div = div_by(us[ic] - us[ic - g.sx], g.Dx[i], g.rDx[i], TWO) +
                       div_by(vs[ic] - vs[ic - g.sy], g.Dy[j], g.rDy[j], TWO) +
                       div_by(ws[ic] - ws[zb], g.Dz[k], g.rDz[k], TWO);
    if (jacobi) {
      b[row] = -row_jp(g, st, i - 2, j - 2, k - 2, row) * ddt * div;
    } else {
      b[row] = -ddt * div;
    }
  }
}

// SPE_matrix::multiply_omp / CSR_matrix::multiply_omp with the reference's entry values
__global__ void __launch_bounds__(kBlock) k_spmv_exact(Geo g, Stencil<double> st, const double *__restrict__ x,
                                                       double *__restrict__ y) {
  for (long long row = blockIdx.x * (long long)kBlock + threadIdx.x; row < g.ncell;
       row += (long long)gridDim.x * kBlock) {
    int ic, jc, kc;
    row_cijk(row, g.nyc, g.nzc, ic, jc, kc);
    y[row] = stencil_row_g(g, st, x, row, ic, jc, kc);
  }
}

// inc/analyses/cfl.hpp:3-78 (get_Cfl) on u*: per cell c = u/Dxs + v/Dys + w/Dzs, each term
// left out on the last face of its own axis (the loops' "-d"), added in that order; the
// maximum of c times dt, and the extremes of each component over its faces.  ss->cfl.
// (The time step computes the same inside k_convdiff_exact; this is the single call.)
__global__ void __launch_bounds__(kBlock) k_cfl(Geo g, double dt, const double *__restrict__ us,
                                                 const double *__restrict__ vs, const double *__restrict__ ws,
                                                 StepCtl sc) {
  const bool two = g.div2 != 0;
  CflAcc cfl;
  for (long long row = blockIdx.x * (long long)kBlock + threadIdx.x; row < g.ncell;
       row += (long long)gridDim.x * kBlock) {
    int i, j, k;
    row_ijk(g, row, i, j, k);
    const long long ic = pidx(g, i, j, k);
    double c = 0.0;
    if (i < g.nx - 3) {
      c += div_by(us[ic], g.Dxs[i], g.rDxs[i], two);
      cfl.comp(0, us[ic]);
    }
    if (j < g.ny - 3) {
      c += div_by(vs[ic], g.Dys[j], g.rDys[j], two);
      cfl.comp(1, vs[ic]);
    }
    if (k < g.nz - 3 + g.pz) {
      c += div_by(ws[ic], g.Dzs[k], g.rDzs[k], two);
      cfl.comp(2, ws[ic]);
    }
    cfl.cell(c);
  }
  cfl_finish(cfl, dt, sc);
}

// Plot3D solution arrays (inc/io/Plot3D/qfile.hpp:62-103) in k-j-i order, i fastest, as
// float32: p, the cell-centred u, v, w (face means, rounded once) and eta
__global__ void __launch_bounds__(kBlock) k_plot3d_pack(Geo g, const double *__restrict__ p,
                                                         const double *__restrict__ u, const double *__restrict__ v,
                                                         const double *__restrict__ w, const double *__restrict__ eta,
                                                         float *__restrict__ out) {
  const long long n = g.ncell;
  for (long long o = blockIdx.x * (long long)kBlock + threadIdx.x; o < n; o += (long long)gridDim.x * kBlock) {
    const int ic = (int)(o % g.nxc);
    const long long r = o / g.nxc;
    const int jc = (int)(r % g.nyc), kc = (int)(r / g.nyc);
    const long long c = pidx(g, ic + 2, jc + 2, kc + 2);
    out[o] = (float)p[c];
    out[n + o] = (float)(0.5 * (u[c - g.sx] + u[c]));
    out[2 * n + o] = (float)(0.5 * (v[c - g.sy] + v[c]));
    out[3 * n + o] = (float)(0.5 * (w[c - 1] + w[c]));
    out[4 * n + o] = (float)eta[c];
  }
}

// QfileRead (inc/io/Plot3D/qfileRead.hpp:66-97): the five cell-centred float32 arrays of a
// .q file (p, u, v, w, eta; i fastest) back to padded fields.  p and eta are copied; u, v, w
// go to faces as the float sum of the cells on both sides, halved in double, and the last
// face of each axis takes its own cell's value.  Interior cells only; eta may be null.
__global__ void __launch_bounds__(kBlock) k_plot3d_unpack(Geo g, const float *__restrict__ in,
                                                           double *__restrict__ p, double *__restrict__ u,
                                                           double *__restrict__ v, double *__restrict__ w,
                                                           double *__restrict__ eta) {
  const long long n = g.ncell, sj = g.nxc, sk = (long long)g.nxc * g.nyc;
  const float *U = in + n, *V = in + 2 * n, *W = in + 3 * n;
  for (long long o = blockIdx.x * (long long)kBlock + threadIdx.x; o < n; o += (long long)gridDim.x * kBlock) {
    const int ic = (int)(o % g.nxc);
    const long long r = o / g.nxc;
    const int jc = (int)(r % g.nyc), kc = (int)(r / g.nyc);
    const long long c = pidx(g, ic + 2, jc + 2, kc + 2);
    p[c] = (double)in[o];
    u[c] = ic == g.nxc - 1 ? (double)U[o] : (double)__fadd_rn(U[o], U[o + 1]) / 2.0;
    v[c] = jc == g.nyc - 1 ? (double)V[o] : (double)__fadd_rn(V[o], V[o + sj]) / 2.0;
    w[c] = kc == g.nzc - 1 ? (double)W[o] : (double)__fadd_rn(W[o], W[o + sk]) / 2.0;
    if (eta) eta[c] = (double)in[4 * n + o];
  }
}

// inc/pressure/Transform.hpp:8-20
__global__ void __launch_bounds__(kBlock) k_transform(Geo g, const double *__restrict__ x, double *__restrict__ p) {
  for (long long row = blockIdx.x * (long long)kBlock + threadIdx.x; row < g.ncell;
       row += (long long)gridDim.x * kBlock) {
    int i, j, k;
    row_ijk(g, row, i, j, k);
    p[pidx(g, i, j, k)] = x[row];
  }
}

// inc/dfib/updateUandF.hpp:90-180 (solid velocity 0), fused with the drag/lift sums of
// virtualF_Int (inc/dfib/virtualForceIntergrator.hpp:67-90) and, in the time step, with
// the part of copyVel (inc/source/copyVel.hpp:4) that matters: the faces update_UandF
// never writes keep the initial values (ui, vi, wi) they hold in the reference's T3.
// One face: T2 = u* - dt dp / Ds, the solid fraction e between the two cells, the forced
// value ec uS + (1 - e) T2 with uS = 0 and the force (nu3 - T2) / dt.  Away from the body
// (eta zero on both sides, all but a few per mille of the faces) e is 0, the forced value T2
// (a negative zero added to ec uS becomes positive) and the force zero: those faces skip the
// FP64 work, the tests on the integer pipe.  A T2 that is not finite takes the general form, so
// that the force carries it to the drag's NaN flag.
__device__ __forceinline__ double uf_face(double T2, double ec, double en, double hf, double dt, double rdt, bool two,
                                          double &force) {
  if (is_zero(ec) && is_zero(en) && finite_int(T2)) {
    force = 0.0;
    return is_zero(T2) ? 0.0 : T2;
  }
  const double e = ec + (en - ec) * hf;
  const double n3 = ec * 0.0 + (1.0 - e) * T2;
  force = div_by(n3 - T2, dt, rdt, two);
  return n3;
}

// 512x256x64: 1.06 -> 0.40 ms (FP64 pipe)
template <bool TWO>
__global__ void __launch_bounds__(kBlock) k_update_uf_exact(
    Geo g, double dt_arg, const double *dtp, int in_step /* step_end mode */, double lz, const double *__restrict__ eta,
    const double *__restrict__ p, const double *__restrict__ us, const double *__restrict__ vs,
    const double *__restrict__ ws, double *__restrict__ u3, double *__restrict__ v3, double *__restrict__ w3,
    double *__restrict__ f, const double *__restrict__ ui, const double *__restrict__ vi,
    const double *__restrict__ wi, double *part, StepScal *ss) {
  const double dt = dtp ? *dtp : dt_arg;
  const bool twot = g.div2t != 0;
  const long long tot = (long long)g.nx * g.ny * g.nz;
  const double rdt = 1.0 / dt;
  double acc[2] = {0.0, 0.0};
  for (long long row = blockIdx.x * (long long)kBlock + threadIdx.x; row < g.ncell;
       row += (long long)gridDim.x * kBlock) {
    int i, j, k;
    row_ijk(g, row, i, j, k);
    const long long ic = pidx(g, i, j, k);
    const double ec = eta[ic], pc = p[ic];
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (i < g.nx - 3) {
      const long long icP = ic + g.sx;
      const double T2u = us[ic] - div_by(dt * (p[icP] - pc), g.Dxs[i], g.rDxs[i], TWO);
      u3[ic] = uf_face(T2u, ec, eta[icP], g.hfx[i], dt, rdt, twot, fx);
      if (f) f[ic] = fx;
    } else if (ui) {
      u3[ic] = ui[ic];
    }
    if (j < g.ny - 3) {
      const long long icP = ic + g.sy;
      const double T2v = vs[ic] - div_by(dt * (p[icP] - pc), g.Dys[j], g.rDys[j], TWO);
      v3[ic] = uf_face(T2v, ec, eta[icP], g.hfy[j], dt, rdt, twot, fy);
      if (f) f[ic + tot] = fy;
    } else if (vi) {
      v3[ic] = vi[ic];
    }
    if (k < g.nz - 3 + g.pz) {  // periodic z: the top face, its upper cell the first one
      const long long icP = (g.pz && k == g.nz - 3) ? ic - (g.nzc - 1) : ic + 1;
      const double T2w = ws[ic] - div_by(dt * (p[icP] - pc), g.Dzs[k], g.rDzs[k], TWO);
      w3[ic] = uf_face(T2w, ec, eta[icP], g.hfz[k], dt, rdt, twot, fz);
      if (f) f[ic + 2 * tot] = fz;
    } else if (wi) {
      w3[ic] = wi[ic];
    }
    if (!is_zero(fx) || !is_zero(fy)) {
      const double vol = g.Dx[i] * g.Dy[j] * g.Dz[k];
      acc[0] += fx * vol;
      acc[1] += fy * vol;
    }
  }
  double out[2];
  if (grid_sum<2>(acc, part, &ss->cnt[0], out) && threadIdx.x == 0) {
    ss->fsum[0] = out[0];
    ss->fsum[1] = out[1];
    ss->cd = -2.0 * out[0] / lz;  // CD_CL, virtualForceIntergrator.hpp:309-314
    ss->cl = -2.0 * out[1] / lz;
    ss->nan_flag = !(isfinite(out[0]) && isfinite(out[1]));
    step_end(ss, dt, in_step);
  }
}

// ---- ghost fill: BC_staggered_main (Boundary_Condition.hpp:37-176) in three phases that
// keep its one-thread order (x faces, then y, then z; each later phase reads cells the
// earlier ones wrote), each fused with the matching part of BC_staggered_copy
// (updateBC.hpp:6-108), whose cells no later phase touches.  bc: Dir/Num table
// (FLOWpassing.hpp:6-40, BcTable).  inlet: optional per-(j,k) inlet velocity taking the
// place of Dir[0][0] (all 1.0 reproduces the reference).
// Two options that are not in the reference: a convective outflow in place of face 1's
// rows (k_outflow_flux first, then k_bc_x), and periodic z in place of faces 4 and 5.

// Convective outflow at the x+ face: d(phi)/dt + Uc d(phi)/dx = 0 for the outlet u face and
// the v, w ghost cells beyond it, implicit upwind in time.  In a step (conv) the outlet u
// before the flux correction is (u_b + cu u_(nx-4)) / (1 + cu), u_b the last step's value
// (the copy in us, which no kernel of the step writes), cu = Uc dt / Dx[nx-3]; at init the
// zero-gradient value u_(nx-4).  The ghosts: (phi_g + cv phi_(nx-3)) / (1 + cv), cv =
// Uc dt / Dxs[nx-3], or phi_(nx-3) at init.
__device__ __forceinline__ double outlet_u(const Geo &g, const double *u, const double *us, double cu, int j,
                                           int k) {
  const double un = u[pidx(g, g.nx - 4, j, k)];
  return us ? (us[pidx(g, g.nx - 3, j, k)] + cu * un) / (1.0 + cu) : un;
}
__device__ __forceinline__ double outlet_ghost(const Geo &g, const double *f, const double *fs, double cv, int j,
                                               int k) {
  const double fn = f[pidx(g, g.nx - 3, j, k)];
  return fs ? (fs[pidx(g, g.nx - 2, j, k)] + cv * fn) / (1.0 + cv) : fn;
}
// cu, cv of a step: dt is the step's (set by the velocity correction's step_end)
__device__ __forceinline__ void outlet_coeffs(const Geo &g, const StepScal *ss, bool conv, double &cu,
                                              double &cv) {
  cu = cv = 0.0;
  if (!conv) return;
  const double dt = ss->dt_step;
  cu = g.uconv * dt / g.Dx[g.nx - 3];
  cv = g.uconv * dt / g.Dxs[g.nx - 3];
}

// The outlet correction: the net flux through the boundary with the outlet faces at
// outlet_u -- inlet u faces, outlet faces, the y-wall v faces and (not periodic) the z-wall
// w faces at the values the ghost fill gives them, each times its face area -- divided by
// the outlet's area, into ss->oflux.  One grid-stride pass over the three face sets.
__global__ void __launch_bounds__(kBlock) k_outflow_flux(Geo g, BcTable t, const double *__restrict__ inlet,
                                                         const double *__restrict__ u, const double *__restrict__ v,
                                                         const double *__restrict__ w, const double *__restrict__ us,
                                                         double *part, StepScal *ss) {
  double cu, cv;
  outlet_coeffs(g, ss, us != nullptr, cu, cv);
  const long long nx_ = g.nyc * (long long)g.nzc, ny_ = g.nxc * (long long)g.nzc,
                  nz_ = g.pz ? 0 : g.nxc * (long long)g.nyc;
  double acc[2] = {0.0, 0.0};  // flux, outlet area
  for (long long q = blockIdx.x * (long long)kBlock + threadIdx.x; q < nx_ + ny_ + nz_;
       q += (long long)gridDim.x * kBlock) {
    if (q < nx_) {
      const int j = (int)(q / g.nzc) + 2, k = (int)(q % g.nzc) + 2;
      const double a = g.Dy[j] * g.Dz[k];
      const double uin = (inlet ? inlet[q] : t.dir[0][0]) + t.num[0][0] * u[pidx(g, 2, j, k)];
      acc[0] += (uin - outlet_u(g, u, us, cu, j, k)) * a;
      acc[1] += a;
    } else if (q < nx_ + ny_) {
      const long long r = q - nx_;
      const int i = (int)(r / g.nzc) + 2, k = (int)(r % g.nzc) + 2;
      const double vb = t.dir[2][1] + t.num[2][1] * v[pidx(g, i, 2, k)];
      const double vt = t.dir[3][1] + t.num[3][1] * v[pidx(g, i, g.ny - 4, k)];
      acc[0] += (vb - vt) * (g.Dx[i] * g.Dz[k]);
    } else {
      const long long r = q - nx_ - ny_;
      const int i = (int)(r / g.nyc) + 2, j = (int)(r % g.nyc) + 2;
      const double wb = t.dir[4][2] + t.num[4][2] * w[pidx(g, i, j, 2)];
      const double wt = t.dir[5][2] + t.num[5][2] * w[pidx(g, i, j, g.nz - 4)];
      acc[0] += (wb - wt) * (g.Dx[i] * g.Dy[j]);
    }
  }
  double out[2];
  if (grid_sum<2>(acc, part, &ss->cnt[8], out) && threadIdx.x == 0) ss->oflux = out[0] / out[1];
}

__global__ void __launch_bounds__(kBlock) k_bc_x(Geo g, BcTable t, const double *__restrict__ inlet, double *u,
                                                 double *v, double *w, double *p, double *us, double *vs, double *ws,
                                                 int do_main, int conv, const StepScal *ss) {
  const int nyc = g.nyc, nzc = g.nzc, nx = g.nx;
  double cu = 0.0, cv = 0.0, corr = 0.0;
  if (do_main && g.outflow) {
    outlet_coeffs(g, ss, conv != 0, cu, cv);
    corr = ss->oflux;
  }
  for (int q = blockIdx.x * kBlock + threadIdx.x; q < nyc * nzc; q += gridDim.x * kBlock) {
    const int j = q / nzc + 2, k = q % nzc + 2;
    auto I = [&](int i) { return pidx(g, i, j, k); };
    if (do_main) {
      const double din = inlet ? inlet[q] : t.dir[0][0];
      u[I(1)] = u[I(0)] = din + t.num[0][0] * u[I(2)];
      v[I(1)] = v[I(0)] = t.dir[0][1] * 2. + (2.0 * t.num[0][1] - 1.0) * v[I(2)];
      w[I(1)] = w[I(0)] = t.dir[0][2] * 2. + (2.0 * t.num[0][2] - 1.0) * w[I(2)];
      if (g.outflow) {
        const double *os = conv ? us : nullptr;
        const double ub = outlet_u(g, u, os, cu, j, k) + corr;
        const double vg = outlet_ghost(g, v, conv ? vs : nullptr, cv, j, k);
        const double wg = outlet_ghost(g, w, conv ? ws : nullptr, cv, j, k);
        u[I(nx - 1)] = u[I(nx - 2)] = u[I(nx - 3)] = ub;
        v[I(nx - 1)] = v[I(nx - 2)] = vg;
        w[I(nx - 1)] = w[I(nx - 2)] = wg;
      } else {
        u[I(nx - 1)] = u[I(nx - 2)] = u[I(nx - 3)] = t.dir[1][0] + t.num[1][0] * u[I(nx - 4)];
        v[I(nx - 1)] = v[I(nx - 2)] = t.dir[1][1] * 2. + (2.0 * t.num[1][1] - 1.0) * v[I(nx - 3)];
        w[I(nx - 1)] = w[I(nx - 2)] = t.dir[1][2] * 2. + (2.0 * t.num[1][2] - 1.0) * w[I(nx - 3)];
      }
      if (p) {
        p[I(1)] = p[I(0)] = p[I(2)];
        p[I(nx - 2)] = p[I(nx - 1)] = p[I(nx - 3)];
      }
    }
    if (us) {
      const int iu[5] = {0, 1, nx - 1, nx - 3, nx - 2};
#pragma unroll
      for (int a = 0; a < 5; ++a) us[I(iu[a])] = u[I(iu[a])];
      const int iv[4] = {0, 1, nx - 2, nx - 1};
#pragma unroll
      for (int a = 0; a < 4; ++a) { vs[I(iv[a])] = v[I(iv[a])]; ws[I(iv[a])] = w[I(iv[a])]; }
    }
  }
}

__global__ void __launch_bounds__(kBlock) k_bc_y(Geo g, BcTable t, double *u, double *v, double *w, double *p,
                                                 double *us, double *vs, double *ws, int do_main) {
  const int nxc = g.nxc, nzc = g.nzc, ny = g.ny;
  for (int q = blockIdx.x * kBlock + threadIdx.x; q < nxc * nzc; q += gridDim.x * kBlock) {
    const int i = q / nzc + 2, k = q % nzc + 2;
    auto J = [&](int j) { return pidx(g, i, j, k); };
    if (do_main) {
      u[J(1)] = u[J(0)] = t.dir[2][0] * 2. + (2.0 * t.num[2][0] - 1.0) * u[J(2)];
      v[J(1)] = v[J(0)] = t.dir[2][1] + t.num[2][1] * v[J(2)];
      w[J(1)] = w[J(0)] = t.dir[2][2] * 2. + (2.0 * t.num[2][2] - 1.0) * w[J(2)];
      v[J(ny - 1)] = v[J(ny - 2)] = v[J(ny - 3)] = t.dir[3][1] + t.num[3][1] * v[J(ny - 4)];
      u[J(ny - 1)] = u[J(ny - 2)] = t.dir[3][0] * 2. + (2.0 * t.num[3][0] - 1.0) * u[J(ny - 3)];
      w[J(ny - 1)] = w[J(ny - 2)] = t.dir[3][2] * 2. + (2.0 * t.num[3][2] - 1.0) * w[J(ny - 3)];
      if (p) {
        p[J(1)] = p[J(0)] = p[J(2)];
        p[J(ny - 2)] = p[J(ny - 1)] = p[J(ny - 3)];
      }
    }
    if (us) {
      const int ju[4] = {0, 1, ny - 2, ny - 1};
#pragma unroll
      for (int a = 0; a < 4; ++a) { us[J(ju[a])] = u[J(ju[a])]; ws[J(ju[a])] = w[J(ju[a])]; }
      const int jv[5] = {0, 1, ny - 3, ny - 2, ny - 1};
#pragma unroll
      for (int a = 0; a < 5; ++a) vs[J(jv[a])] = v[J(jv[a])];
    }
  }
}

// periodic z: the two ghost layers on each side take the images nzc cells away (w's face
// 1 is the image of the top face nz-3), over the whole padded (i, j) plane so that the
// edges and corners next to the z ghosts are periodic too; the copy into T1 as the
// reference's (interior (i, j), the z ghosts and w's face nz-3)
// (grids of fewer than four cells along z: their ghosts are each other's images)
__global__ void __launch_bounds__(kBlock) k_bc_zp_thin(Geo g, double *u, double *v, double *w, double *p, double *us,
                                                       double *vs, double *ws, int do_main) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  for (int q = blockIdx.x * kBlock + threadIdx.x; q < nx * ny; q += gridDim.x * kBlock) {
    const int i = q / ny, j = q % ny;
    const long long base = pidx(g, i, j, 0);
    if (do_main) {
      double *f[4] = {u, v, w, p};
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        if (!f[a]) continue;
        f[a][base + 0] = f[a][base + nz - 4];
        f[a][base + 1] = f[a][base + nz - 3];
        f[a][base + nz - 2] = f[a][base + 2];
        f[a][base + nz - 1] = f[a][base + 3];
      }
    }
    if (us && i >= 2 && i < nx - 2 && j >= 2 && j < ny - 2) {
      const int ku[4] = {0, 1, nz - 2, nz - 1};
#pragma unroll
      for (int a = 0; a < 4; ++a) { us[base + ku[a]] = u[base + ku[a]]; vs[base + ku[a]] = v[base + ku[a]]; }
      const int kw[5] = {0, 1, nz - 3, nz - 2, nz - 1};
#pragma unroll
      for (int a = 0; a < 5; ++a) ws[base + kw[a]] = w[base + kw[a]];
    }
  }
}

// The same from four cells on: every source value first, so that the loads of all fields are in
// flight together (written field by field each store held the next load back), and two values a
// request where the lines are 16-byte aligned (PAIR: an even nz): 512x256x64 66 -> 43 us
template <bool PAIR>
__global__ void __launch_bounds__(kBlock) k_bc_zp(Geo g, double *__restrict__ u, double *__restrict__ v,
                                                  double *__restrict__ w, double *__restrict__ p,
                                                  double *__restrict__ us, double *__restrict__ vs,
                                                  double *__restrict__ ws, int do_main) {
  auto ld = [](const double *f) { return PAIR ? *reinterpret_cast<const double2 *>(f) : make_double2(f[0], f[1]); };
  auto st = [](double *f, double2 a) {
    if (PAIR) {
      *reinterpret_cast<double2 *>(f) = a;
    } else {
      f[0] = a.x;
      f[1] = a.y;
    }
  };
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  // where the ghosts' values stand: the images, or (no main part) the ghosts themselves
  const int sl = do_main ? nz - 4 : 0, sh = do_main ? 2 : nz - 2;
  for (int q = blockIdx.x * kBlock + threadIdx.x; q < nx * ny; q += gridDim.x * kBlock) {
    const int i = q / ny, j = q % ny;
    const long long b = pidx(g, i, j, 0);
    const bool copy = us && i >= 2 && i < nx - 2 && j >= 2 && j < ny - 2;
    if (!do_main && !copy) continue;
    const double2 ul = ld(u + b + sl), uh = ld(u + b + sh), vl = ld(v + b + sl), vh = ld(v + b + sh);
    const double2 wl = ld(w + b + sl), wh = ld(w + b + sh);
    const double wt = copy ? w[b + nz - 3] : 0.0;
    if (do_main) {
      if (p) {
        const double2 pl = ld(p + b + sl), ph = ld(p + b + sh);
        st(p + b, pl);
        st(p + b + nz - 2, ph);
      }
      st(u + b, ul);
      st(u + b + nz - 2, uh);
      st(v + b, vl);
      st(v + b + nz - 2, vh);
      st(w + b, wl);
      st(w + b + nz - 2, wh);
    }
    if (copy) {
      st(us + b, ul);
      st(us + b + nz - 2, uh);
      st(vs + b, vl);
      st(vs + b + nz - 2, vh);
      st(ws + b, wl);
      st(ws + b + nz - 2, wh);
      ws[b + nz - 3] = wt;
    }
  }
}

// (PAIR: an even nz and 16-byte aligned fields, two values a store; 512x256x64 55 -> 42 us)
template <bool PAIR>
__global__ void __launch_bounds__(kBlock) k_bc_z(Geo g, BcTable t, double *__restrict__ u, double *__restrict__ v,
                                                 double *__restrict__ w, double *__restrict__ p,
                                                 double *__restrict__ us, double *__restrict__ vs,
                                                 double *__restrict__ ws, int do_main) {
  auto both = [](double *f, double x, double y) {
    if (PAIR) {
      *reinterpret_cast<double2 *>(f) = make_double2(x, y);
    } else {
      f[0] = x;
      f[1] = y;
    }
  };
  const int nxc = g.nxc, nyc = g.nyc, nz = g.nz;
  for (int q = blockIdx.x * kBlock + threadIdx.x; q < nxc * nyc; q += gridDim.x * kBlock) {
    const int i = q / nyc + 2, j = q % nyc + 2;
    const long long base = pidx(g, i, j, 0);
    if (do_main) {
      // every source value first (each line's ends lie 8 B x nz apart: the loads of all
      // four fields are in flight together), then the ghosts
      const double u2 = u[base + 2], v2 = v[base + 2], w2 = w[base + 2];
      const double uT = u[base + nz - 3], vT = v[base + nz - 3], wT = w[base + nz - 4];
      const double p2 = p ? p[base + 2] : 0.0, pT = p ? p[base + nz - 3] : 0.0;
      const double ub = t.dir[4][0] * 2. + (2.0 * t.num[4][0] - 1.0) * u2;
      const double vb = t.dir[4][1] * 2. + (2.0 * t.num[4][1] - 1.0) * v2;
      const double wb = t.dir[4][2] + t.num[4][2] * w2;
      const double wt = t.dir[5][2] + t.num[5][2] * wT;
      const double ut = t.dir[5][0] * 2. + (2.0 * t.num[5][0] - 1.0) * uT;
      const double vt = t.dir[5][1] * 2. + (2.0 * t.num[5][1] - 1.0) * vT;
      both(u + base, ub, ub);
      both(v + base, vb, vb);
      both(w + base, wb, wb);
      w[base + nz - 3] = wt;
      both(w + base + nz - 2, wt, wt);
      both(u + base + nz - 2, ut, ut);
      both(v + base + nz - 2, vt, vt);
      if (p) {
        both(p + base, p2, p2);
        both(p + base + nz - 2, pT, pT);
      }
      if (us) {  // the copies of what this thread just wrote
        both(us + base, ub, ub);
        both(us + base + nz - 2, ut, ut);
        both(vs + base, vb, vb);
        both(vs + base + nz - 2, vt, vt);
        both(ws + base, wb, wb);
        ws[base + nz - 3] = wt;
        both(ws + base + nz - 2, wt, wt);
      }
      continue;
    }
    if (us) {
      const int ku[4] = {0, 1, nz - 2, nz - 1};
#pragma unroll
      for (int a = 0; a < 4; ++a) { us[base + ku[a]] = u[base + ku[a]]; vs[base + ku[a]] = v[base + ku[a]]; }
      const int kw[5] = {0, 1, nz - 3, nz - 2, nz - 1};
#pragma unroll
      for (int a = 0; a < 5; ++a) ws[base + kw[a]] = w[base + kw[a]];
    }
  }
}

// inc/dfib/setEta.hpp:136-198: per (i,j) column, solid fraction at k = 0 by 100x100
// sub-sampling of cells within half a cell diagonal of the circle.  One warp per column:
// the lanes split the 100 sub-rows and the warp adds their integer counts (exact in any
// order), so a band column costs 400 sample tests per lane instead of 10000 in one thread.
__global__ void __launch_bounds__(kBlock) k_eta_plane(Geo g, const double *__restrict__ X,
                                                      const double *__restrict__ Y, double cx, double cy,
                                                      double R, double *__restrict__ eta) {
  const int nxc = g.nxc, nyc = g.nyc;
  const int lane = threadIdx.x & 31, wpb = kBlock / 32;
  for (long long q = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); q < (long long)nxc * nyc;
       q += (long long)gridDim.x * wpb) {
    const int i = (int)(q / nyc) + 2, j = (int)(q % nyc) + 2;
    const long long icel = pidx(g, i, j, 0);
    const double Diagonal = sqrt(g.Dx[i] * g.Dx[i] + g.Dy[j] * g.Dy[j]) * 0.5;
    const double ddx = ((X[i] + X[i + 1]) * 0.5) - cx;
    const double ddy = ((Y[j] + Y[j + 1]) * 0.5) - cy;
    const double Distance = sqrt(ddx * ddx + ddy * ddy);
    if (fabs(Distance - R) < Diagonal) {
      const int nsub = 100;
      const double dyg = g.Dy[j] / (double)nsub;
      const double dxg = g.Dx[i] / (double)nsub;
      unsigned xi = 0;
      for (int ii = lane; ii < nsub; ii += 32) {
        const double sx0 = X[i] + (double)ii * dxg, sx1 = X[i] + (double)(ii + 1) * dxg;
        const double a = (sx0 + sx1) * 0.5 - cx;
        for (int jj = 0; jj < nsub; ++jj) {
          const double sy0 = Y[j] + (double)jj * dyg, sy1 = Y[j] + (double)(jj + 1) * dyg;
          const double b = (sy0 + sy1) * 0.5 - cy;
          if (sqrt(a * a + b * b) <= R) ++xi;
        }
      }
      xi = __reduce_add_sync(0xffffffffu, xi);
      if (lane == 0) eta[icel] = (double)xi * (1.0 / ((double)nsub * (double)nsub));
    } else if (lane == 0) {
      eta[icel] = Distance > R ? 0. : 1.;
    }
  }
}

// setEta.hpp:200-203: copy plane k = 0 to k in [1, nz-1) for i < nx-1, j < ny-1
__global__ void __launch_bounds__(kBlock) k_eta_extrude(Geo g, double *__restrict__ eta) {
  const long long n = (long long)(g.nx - 1) * (g.ny - 1) * (g.nz - 2);
  for (long long q = blockIdx.x * (long long)kBlock + threadIdx.x; q < n; q += (long long)gridDim.x * kBlock) {
    const int k = (int)(q % (g.nz - 2)) + 1;
    const long long ij = q / (g.nz - 2);
    const int j = (int)(ij % (g.ny - 1)), i = (int)(ij / (g.ny - 1));
    eta[pidx(g, i, j, k)] = eta[pidx(g, i, j, 0)];
  }
}

// ---- launchers ----
constexpr size_t kQuickSmem = 24 * sizeof(double);  // shared memory of k_convdiff_quick per thread
bool convdiff_prepare() {
  const int most = (int)kQuickSmem * 512;  // above the default 48 KB
  const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
  return cudaFuncSetAttribute(k_convdiff_quick<false, false>, a, most) == cudaSuccess &&
         cudaFuncSetAttribute(k_convdiff_quick<false, true>, a, most) == cudaSuccess &&
         cudaFuncSetAttribute(k_convdiff_quick<true, false>, a, most) == cudaSuccess &&
         cudaFuncSetAttribute(k_convdiff_quick<true, true>, a, most) == cudaSuccess;
}
template <bool AB>
static void convdiff_exact(cudaStream_t s, int nblk, const Geo &g, int scheme, double dt, double nu, const double *nut,
                           const double *u, const double *v, const double *w, double *us, double *vs, double *ws,
                           const StepCtl &sc) {
  if (scheme == CFDGB_LUD)
    k_convdiff_exact<CFDGB_LUD, AB><<<nblk, kBlock, 0, s>>>(g, dt, nu, nut, u, v, w, us, vs, ws, sc);
  else if (scheme == CFDGB_UD)
    k_convdiff_exact<CFDGB_UD, AB><<<nblk, kBlock, 0, s>>>(g, dt, nu, nut, u, v, w, us, vs, ws, sc);
  else {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const QuickPlan pl = quick_plan(g, nsm);
    const size_t smem = kQuickSmem * (size_t)pl.threads;
    const dim3 grid(pl.gx, pl.gy, pl.gz);
    if (g.div2)
      k_convdiff_quick<AB, true><<<grid, pl.threads, smem, s>>>(g, pl, dt, nu, nut, u, v, w, us, vs, ws, sc);
    else
      k_convdiff_quick<AB, false><<<grid, pl.threads, smem, s>>>(g, pl, dt, nu, nut, u, v, w, us, vs, ws, sc);
  }
}
void launch_convdiff_exact(cudaStream_t s, int nblk, const Geo &g, int scheme, double dt, double nu,
                           const double *nut, const double *u, const double *v, const double *w, double *us,
                           double *vs, double *ws, const StepCtl &sc) {
  if (sc.time_order > 1)
    convdiff_exact<true>(s, nblk, g, scheme, dt, nu, nut, u, v, w, us, vs, ws, sc);
  else
    convdiff_exact<false>(s, nblk, g, scheme, dt, nu, nut, u, v, w, us, vs, ws, sc);
}
void launch_smagorinsky(cudaStream_t s, int nblk, const Geo &g, const double *l2, const double *u, const double *v,
                        const double *w, double *nut) {
  k_smagorinsky<<<nblk, kBlock, 0, s>>>(g, l2, u, v, w, nut);
}
void launch_rhs_exact(cudaStream_t s, int nblk, const Geo &g, double dt, const double *dtp, const double *us,
                      const double *vs, const double *ws, int jacobi, const Stencil<double> &st, double *b) {
  (g.div2 ? k_rhs_exact<true> : k_rhs_exact<false>)<<<nblk, kBlock, 0, s>>>(g, dt, dtp, us, vs, ws, jacobi, st, b);
}
void launch_spmv_exact(cudaStream_t s, int nblk, const Geo &g, const Stencil<double> &st, const double *x,
                       double *y) {
  k_spmv_exact<<<nblk, kBlock, 0, s>>>(g, st, x, y);
}
void launch_cfl(cudaStream_t s, int nblk, const Geo &g, double dt, const double *us, const double *vs,
                const double *ws, double *part, StepScal *ss) {
  StepCtl sc{};
  sc.ss = ss;
  sc.part = part;
  k_cfl<<<nblk, kBlock, 0, s>>>(g, dt, us, vs, ws, sc);
}
void launch_plot3d_pack(cudaStream_t s, int nblk, const Geo &g, const double *p, const double *u, const double *v,
                        const double *w, const double *eta, float *out) {
  k_plot3d_pack<<<nblk, kBlock, 0, s>>>(g, p, u, v, w, eta, out);
}
void launch_plot3d_unpack(cudaStream_t s, int nblk, const Geo &g, const float *in, double *p, double *u, double *v,
                          double *w, double *eta) {
  k_plot3d_unpack<<<nblk, kBlock, 0, s>>>(g, in, p, u, v, w, eta);
}
void launch_transform(cudaStream_t s, int nblk, const Geo &g, const double *x, double *p) {
  k_transform<<<nblk, kBlock, 0, s>>>(g, x, p);
}
void launch_update_uf_exact(cudaStream_t s, int nblk, const Geo &g, double dt, const double *dtp, int step_mode,
                            double lz, const double *eta, const double *p, const double *us, const double *vs,
                            const double *ws, double *u3, double *v3, double *w3, double *f, const double *ui,
                            const double *vi, const double *wi, double *part, StepScal *ss) {
  (g.div2 ? k_update_uf_exact<true> : k_update_uf_exact<false>)<<<nblk, kBlock, 0, s>>>(
      g, dt, dtp, step_mode, lz, eta, p, us, vs, ws, u3, v3, w3, f, ui, vi, wi, part, ss);
}
void launch_bc(cudaStream_t s, const Geo &g, double *u, double *v, double *w, double *p, double *us,
               double *vs, double *ws, int do_main, const double *inlet, int conv, double *part, StepScal *ss,
               int nblk) {
  const BcTable t = flowpassing_table(g.walls);
  auto blocks = [](long long n) { return (int)((n + kBlock - 1) / kBlock < 1024 ? (n + kBlock - 1) / kBlock : 1024); };
  conv = conv && us;  // the last step's outlet values live in T1
  if (do_main && g.outflow) {
    const long long nf = (long long)g.nyc * g.nzc + (long long)g.nxc * g.nzc + (g.pz ? 0LL : (long long)g.nxc * g.nyc);
    const int fb = (int)std::min<long long>((nf + kBlock - 1) / kBlock, (long long)nblk);
    k_outflow_flux<<<fb, kBlock, 0, s>>>(g, t, inlet, u, v, w, conv ? us : nullptr, part, ss);
  }
  k_bc_x<<<blocks((long long)g.nyc * g.nzc), kBlock, 0, s>>>(g, t, inlet, u, v, w, p, us, vs, ws, do_main, conv, ss);
  k_bc_y<<<blocks((long long)g.nxc * g.nzc), kBlock, 0, s>>>(g, t, u, v, w, p, us, vs, ws, do_main);
  uintptr_t at = 0;
  for (const double *f : {u, v, w, p, us, vs, ws}) at |= reinterpret_cast<uintptr_t>(f);
  const bool pair = g.nz % 2 == 0 && at % 16 == 0;
  if (g.pz)
    (g.nzc < 4 ? k_bc_zp_thin : pair ? k_bc_zp<true> : k_bc_zp<false>)<<<blocks((long long)g.nx * g.ny), kBlock, 0, s>>>(
        g, u, v, w, p, us, vs, ws, do_main);
  else
    (pair ? k_bc_z<true> : k_bc_z<false>)<<<blocks((long long)g.nxc * g.nyc), kBlock, 0, s>>>(g, t, u, v, w, p, us, vs,
                                                                                           ws, do_main);
}
void launch_eta(cudaStream_t s, int nblk, const Geo &g, const double *X, const double *Y, double cx, double cy,
                double R, double *eta) {
  const long long cols = (long long)g.nxc * g.nyc;
  const int wpb = kBlock / 32;
  const int blocks = (int)std::min<long long>((cols + wpb - 1) / wpb, 65535LL * 8);
  k_eta_plane<<<blocks, kBlock, 0, s>>>(g, X, Y, cx, cy, R, eta);
  k_eta_extrude<<<nblk, kBlock, 0, s>>>(g, eta);
}

}  // namespace cfdgb

// ---- self-check of div_by against IEEE division (this file is built with -prec-div=true) ----
namespace cfdgb {
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__global__ void __launch_bounds__(kBlock) k_check_div(long long n, unsigned long long seed, double b, double y,
                                                      bool two, unsigned long long *bad) {
  unsigned long long miss = 0;
  for (long long q = blockIdx.x * (long long)kBlock + threadIdx.x; q < n; q += (long long)gridDim.x * kBlock) {
    const unsigned long long h1 = mix64(seed ^ (unsigned long long)q), h2 = mix64(h1);
    double a;
    if (q % 1000 == 0) {
      a = (q % 2000 == 0) ? 0.0 : -0.0;
    } else if (q % 10 == 0) {
      a = b * (double)(long long)(h2 % 1000000);  // exact quotients
    } else {
      const double m = 1.0 + (double)(h1 >> 12) * 0x1.0p-52;  // [1, 2), 52 random bits
      a = scalbn(m, (int)(h2 % 81) - 40) * ((h2 >> 40) & 1 ? -1.0 : 1.0);
    }
    if (__double_as_longlong(a / b) != __double_as_longlong(div_by(a, b, y, two))) ++miss;
  }
  if (miss) atomicAdd(bad, miss);
}
}  // namespace cfdgb

extern "C" int cfdgb_check_division(long long n, uint64_t seed, double b, unsigned long long *mismatches) {
  using namespace cfdgb;
  if (!mismatches || n < 0 || !(b != 0.0) || !std::isfinite(b)) return CFDGB_EINVAL;
  unsigned long long *d = nullptr;
  if (cudaMalloc(&d, sizeof(*d)) != cudaSuccess) return CFDGB_ECUDA;
  cudaMemset(d, 0, sizeof(*d));
  // the form the library uses for a context whose only divisor is b
  k_check_div<<<1216, kBlock>>>(n, seed, b, 1.0 / b, !div_certified(b), d);
  const cudaError_t e = cudaMemcpy(mismatches, d, sizeof(*d), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? CFDGB_OK : CFDGB_ECUDA;
}
