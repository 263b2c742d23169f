// Geometric multigrid V-cycle in FP32: the preconditioner of the FP32 BiCGSTAB sweep
// inside the FP64 refinement (the reference has no multigrid; its Poisson operator on a
// uniform grid is the 7-point Neumann Laplacian of SPE_sparseMatrix.hpp:42-85, which every
// level here rediscretises at its own spacing).
//
// Cell-centred hierarchy: a coarse cell is the union of 2 cells along each halved axis.
// Restriction averages the fine residual over a coarse cell's children; prolongation is
// the cell-centred trilinear interpolation (weights 3/4 and 1/4 per halved axis, the
// parent's value standing in for a neighbour beyond a Neumann wall, the wrapped cell
// across a periodic z end); the smoother is
// red-black Gauss-Seidel, one sweep before and one after the coarse correction; the
// coarsest level (at most kMgSharedCells cells) is solved by red-black sweeps in the
// shared memory of one block.  The V-cycle is a fixed linear map, as a right
// preconditioner of BiCGSTAB requires.  Every kernel is pointwise or a stencil over one
// level and reads sc->done first, so a captured chunk of iterations idles once the sweep
// has stopped.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "cfdgb_internal.cuh"
#include "kernels.h"

namespace cfdgb {

// Programmatic dependent launch (griddepcontrol): a V-cycle kernel is launched so that it
// may be scheduled while its predecessor finishes.  It waits for the predecessor's
// completion and memory (pdl_wait) before reading anything, and lets its successor be
// scheduled once its own results are stored (pdl_trigger); a block that returns early
// counts as triggered.  The small levels' kernels are launch-latency-bound.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

#define FOR_LEVEL(L)                                   \
  const int k = blockIdx.x * blockDim.x + threadIdx.x; \
  const int j = blockIdx.y * blockDim.y + threadIdx.y; \
  const bool on_ = (k < (L).nz) && (j < (L).ny);       \
  for (int i = blockIdx.z; on_ && i < (L).nx; i += gridDim.z)

template <typename T>
__device__ __forceinline__ long long lrow(const MgLevelT<T> &L, int i, int j, int k) {
  return ((long long)i * L.ny + j) * L.nz + k;
}

// Rounded operations the compiler does not contract: the quad smoother, the pair transfers
// and the marching kernels form each value by the same explicit sequence, so that they give
// identical results.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
// wx a + wy e + wz f (the weighted neighbour sums of lnb's three axes)
template <typename T>
__device__ __forceinline__ T wsum(const MgLevelT<T> &L, T a, T e, T f) {
  return fma_rn(L.wz, f, fma_rn(L.wy, e, mul_rn(L.wx, a)));
}
// one child's residual b - d x + (neighbour sum), b already scaled
template <typename T>
__device__ __forceinline__ T resid(T bb, T d, T x, T nb) { return add_rn(fma_rn(-d, x, bb), nb); }

// z neighbours of a cell: those that exist (Neumann), or both across the wrap (periodic z,
// none on a level one cell thick, whose wrapped neighbours are the cell itself)
template <typename T>
__device__ __forceinline__ int zcount(const MgLevelT<T> &L, int k) {
  return L.pz ? (L.nz > 1 ? 2 : 0) : (k > 0) + (k < L.nz - 1);
}

// diagonal of a row: the weights of the neighbours that exist
template <typename T>
__device__ __forceinline__ T ldiag(const MgLevelT<T> &L, int i, int j, int k) {
  return L.wx * (T)((i > 0) + (i < L.nx - 1)) + L.wy * (T)((j > 0) + (j < L.ny - 1)) + L.wz * (T)zcount(L, k);
}

// 1/diag of the row (ldiag's reciprocal, from the level's table)
template <typename T>
__device__ __forceinline__ T linv(const MgLevelT<T> &L, int i, int j, int k) {
  return L.idg[9 * ((i > 0) + (i < L.nx - 1)) + 3 * ((j > 0) + (j < L.ny - 1)) + zcount(L, k)];
}

// weighted sum of the neighbours' values (minus the off-diagonal part of the row)
template <typename T>
__device__ __forceinline__ T lnb(const MgLevelT<T> &L, const T *x, int i, int j, int k, long long r) {
  const long long sx = (long long)L.ny * L.nz;
  T a = T(0), b = T(0), c = T(0);
  if (i > 0) a += x[r - sx];
  if (i < L.nx - 1) a += x[r + sx];
  if (j > 0) b += x[r - L.nz];
  if (j < L.ny - 1) b += x[r + L.nz];
  if (L.pz) {
    if (L.nz > 1) {
      c += x[k > 0 ? r - 1 : r + L.nz - 1];
      c += x[k < L.nz - 1 ? r + 1 : r + 1 - L.nz];
    }
  } else {
    if (k > 0) c += x[r - 1];
    if (k < L.nz - 1) c += x[r + 1];
  }
  return L.wx * a + L.wy * b + L.wz * c;
}

// One colour of a red-black Gauss-Seidel sweep (colour = (i + j + k) & 1).  zero: x starts
// at zero, so the cells of this colour take b / diag and the others are set to zero.
// bscale: b holds Jacobi-scaled rows (b / diag), which are unscaled first.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_mg_smooth(MgLevelT<T> L, int colour, int zero, int bscale,
                                                      const T *__restrict__ b, T *x, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  FOR_LEVEL(L) {
    const long long r = lrow(L, i, j, k);
    if (((i + j + k) & 1) != colour) {
      if (zero) x[r] = T(0);
      continue;
    }
    T bb = b[r];
    if (bscale) bb *= ldiag(L, i, j, k);
    const T num = zero ? bb : bb + lnb(L, x, i, j, k, r);
    x[r] = num * linv(L, i, j, k);
  }
}

// The same colour pass on quads of four consecutive k cells (nz % 4 == 0): a thread updates
// the two cells of the colour in its quad and stores the whole quad, the other two
// unchanged (no thread writes them in this pass, so rewriting them races with nothing).
// 3-D launch (quads along x, rows along y, planes strided over z: no index division), the
// row's neighbour counts along x and y taken once per quad.  Neighbour sums in the order
// of lnb, diagonals as ldiag / linv form them.
__global__ void __launch_bounds__(kBlock) k_mg_smooth4(MgLevel L, int colour, int zero, int bscale,
                                                       const float *__restrict__ b, float *x, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  const int kq = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (kq >= (L.nz >> 2) || j >= L.ny) return;  // no barrier below
  const long long sx = (long long)L.ny * L.nz;
  const int k0 = 4 * kq;
  const bool jm = j > 0, jp = j < L.ny - 1;
  const int cy = (int)jm + (int)jp;
  int cz[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) cz[c] = zcount(L, k0 + c);
  for (int i = blockIdx.z; i < L.nx; i += gridDim.z) {
    const long long r = lrow(L, i, j, k0);
    const bool im = i > 0, ip = i < L.nx - 1;
    const int cx = (int)im + (int)ip, cxy = 9 * cx + 3 * cy;
    const float dxy = L.wx * (float)cx + L.wy * (float)cy;  // ldiag's first two terms, in its order
    const int t0 = (i + j + k0 + colour) & 1;  // first cell of the colour in the quad
    const float4 bq = *reinterpret_cast<const float4 *>(b + r);
    const float bv[4] = {bq.x, bq.y, bq.z, bq.w};
    float o[4];
    if (zero) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if ((c & 1) != t0) {
          o[c] = 0.f;
          continue;
        }
        const float bb = bscale ? mul_rn(bv[c], dxy + L.wz * (float)cz[c]) : bv[c];
        o[c] = mul_rn(bb, L.idg[cxy + cz[c]]);
      }
    } else {
      const float4 xq = *reinterpret_cast<const float4 *>(x + r);
      const float xv[4] = {xq.x, xq.y, xq.z, xq.w};
      const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 xm = im ? *reinterpret_cast<const float4 *>(x + r - sx) : z4;
      const float4 xp = ip ? *reinterpret_cast<const float4 *>(x + r + sx) : z4;
      const float4 ym = jm ? *reinterpret_cast<const float4 *>(x + r - L.nz) : z4;
      const float4 yp = jp ? *reinterpret_cast<const float4 *>(x + r + L.nz) : z4;
      const float xmv[4] = {xm.x, xm.y, xm.z, xm.w}, xpv[4] = {xp.x, xp.y, xp.z, xp.w};
      const float ymv[4] = {ym.x, ym.y, ym.z, ym.w}, ypv[4] = {yp.x, yp.y, yp.z, yp.w};
      // the cells left and right of the quad (periodic z: across the wrap)
      const float kl = k0 > 0 ? x[r - 1] : (L.pz ? x[r + L.nz - 1] : 0.f);
      const float kr = k0 + 4 < L.nz ? x[r + 4] : (L.pz ? x[r + 4 - L.nz] : 0.f);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        o[c] = xv[c];
        if ((c & 1) != t0) continue;
        const int k = k0 + c;
        float a = 0.f, e = 0.f, f = 0.f;
        if (im) a += xmv[c];
        if (ip) a += xpv[c];
        if (jm) e += ymv[c];
        if (jp) e += ypv[c];
        if (k > 0 || L.pz) f += c == 0 ? kl : xv[c - 1];
        if (k < L.nz - 1 || L.pz) f += c == 3 ? kr : xv[c + 1];
        const float bb = bscale ? mul_rn(bv[c], dxy + L.wz * (float)cz[c]) : bv[c];
        o[c] = mul_rn(add_rn(bb, wsum(L, a, e, f)), L.idg[cxy + cz[c]]);
      }
    }
    *reinterpret_cast<float4 *>(x + r) = make_float4(o[0], o[1], o[2], o[3]);
  }
}

// bc = average over each coarse cell's children of the fine residual b - A x
template <typename T>
__global__ void __launch_bounds__(kBlock) k_mg_restrict(MgLevelT<T> F, MgLevelT<T> Cl, int bscale,
                                                        const T *__restrict__ bf, const T *__restrict__ xf,
                                                        T *__restrict__ bc, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  const T inv = T(1) / (T)(F.fx * F.fy * F.fz);
  FOR_LEVEL(Cl) {
    T sum = T(0);
    for (int a = 0; a < F.fx; ++a)
      for (int e = 0; e < F.fy; ++e)
        for (int c = 0; c < F.fz; ++c) {
          const int fi = i * F.fx + a, fj = j * F.fy + e, fk = k * F.fz + c;
          const long long r = lrow(F, fi, fj, fk);
          const T d = ldiag(F, fi, fj, fk);
          T bb = bf[r];
          if (bscale) bb *= d;
          sum += bb - d * xf[r] + lnb(F, xf, fi, fj, fk, r);
        }
    bc[lrow(Cl, i, j, k)] = sum * inv;
  }
}

// the two coarse cells a fine cell interpolates from along one axis, and their weights;
// per: the axis is periodic
template <typename T>
__device__ __forceinline__ void axis_taps(int i, int f, int n, int (&c)[2], T (&w)[2], bool per = false) {
  if (f == 1) {
    c[0] = c[1] = i;
    w[0] = T(1);
    w[1] = T(0);
    return;
  }
  const int p = i >> 1;
  int q = p + ((i & 1) ? 1 : -1);
  // beyond a wall: the parent's value (zero normal gradient); periodic: the wrapped cell
  if (q < 0 || q >= n) q = per ? (q + n) % n : p;
  c[0] = p;
  c[1] = q;
  w[0] = T(0.75);
  w[1] = T(0.25);
}

// (P xc) at fine cell (i, j, k): cell-centred trilinear interpolation
template <typename T>
__device__ __forceinline__ T prolong_at(const MgLevelT<T> &F, const MgLevelT<T> &Cl, const T *__restrict__ xc, int i,
                                        int j, int k) {
  int ci[2], cj[2], ck[2];
  T wi[2], wj[2], wk[2];
  axis_taps(i, F.fx, Cl.nx, ci, wi);
  axis_taps(j, F.fy, Cl.ny, cj, wj);
  axis_taps(k, F.fz, Cl.nz, ck, wk, F.pz != 0);
  T v = T(0);
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const T w = wi[a] * wj[e] * wk[c];
        if (w != T(0)) v += w * xc[lrow(Cl, ci[a], cj[e], ck[c])];
      }
  return v;
}

// xf += P xc
template <typename T>
__global__ void __launch_bounds__(kBlock) k_mg_prolong(MgLevelT<T> F, MgLevelT<T> Cl, const T *__restrict__ xc,
                                                       T *__restrict__ xf, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  FOR_LEVEL(F) {
    xf[lrow(F, i, j, k)] += prolong_at(F, Cl, xc, i, j, k);
  }
}

// ---- transfers when every axis halves (fx = fy = fz = 2): one thread per coarse cell,
// its eight children loaded once (pairs along k as one vector load) and their neighbours
// shared, the arithmetic and summation order of k_mg_restrict / k_mg_prolong ----
template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };
template <typename T>
__device__ __forceinline__ void ld2(const T *p, T &a, T &b) {
  const typename Vec2<T>::type v = *reinterpret_cast<const typename Vec2<T>::type *>(p);
  a = v.x;
  b = v.y;
}
template <typename T>
__device__ __forceinline__ void st2(T *p, T a, T b) {
  typename Vec2<T>::type v;
  v.x = a;
  v.y = b;
  *reinterpret_cast<typename Vec2<T>::type *>(p) = v;
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_mg_restrict8(MgLevelT<T> F, MgLevelT<T> Cl, int bscale,
                                                         const T *__restrict__ bf, const T *__restrict__ xf,
                                                         T *__restrict__ bc, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  const T inv = T(1) / T(8);
  const long long sx = (long long)F.ny * F.nz, sy = F.nz;
  FOR_LEVEL(Cl) {
    const int i0 = 2 * i, j0 = 2 * j, k0 = 2 * k;
    const long long r0 = lrow(F, i0, j0, k0);
    T xv[2][2][2], bv[2][2][2], xim[2][2], xip[2][2], xjm[2][2], xjp[2][2], xkm[2][2], xkp[2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const long long r = r0 + a * sx + e * sy;
        ld2(xf + r, xv[a][e][0], xv[a][e][1]);
        ld2(bf + r, bv[a][e][0], bv[a][e][1]);
        xkm[a][e] = k0 > 0 ? xf[r - 1] : (F.pz ? xf[r + F.nz - 1] : T(0));
        xkp[a][e] = k0 + 2 < F.nz ? xf[r + 2] : (F.pz ? xf[r + 2 - F.nz] : T(0));
      }
#pragma unroll
    for (int e = 0; e < 2; ++e) {  // x neighbours of the i0 and i0+1 planes
      if (i0 > 0) ld2(xf + r0 - sx + e * sy, xim[e][0], xim[e][1]);
      else xim[e][0] = xim[e][1] = T(0);
      if (i0 + 2 < F.nx) ld2(xf + r0 + 2 * sx + e * sy, xip[e][0], xip[e][1]);
      else xip[e][0] = xip[e][1] = T(0);
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {  // y neighbours
      if (j0 > 0) ld2(xf + r0 + a * sx - sy, xjm[a][0], xjm[a][1]);
      else xjm[a][0] = xjm[a][1] = T(0);
      if (j0 + 2 < F.ny) ld2(xf + r0 + a * sx + 2 * sy, xjp[a][0], xjp[a][1]);
      else xjp[a][0] = xjp[a][1] = T(0);
    }
    T sum = T(0);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int fi = i0 + a, fj = j0 + e, fk = k0 + c;
          T ax = T(0), ay = T(0), az = T(0);  // lnb's terms in its order
          if (fi > 0) ax += a ? xv[0][e][c] : xim[e][c];
          if (fi < F.nx - 1) ax += a ? xip[e][c] : xv[1][e][c];
          if (fj > 0) ay += e ? xv[a][0][c] : xjm[a][c];
          if (fj < F.ny - 1) ay += e ? xjp[a][c] : xv[a][1][c];
          if (fk > 0 || F.pz) az += c ? xv[a][e][0] : xkm[a][e];
          if (fk < F.nz - 1 || F.pz) az += c ? xkp[a][e] : xv[a][e][1];
          const T d = ldiag(F, fi, fj, fk);
          const T bb = bscale ? mul_rn(bv[a][e][c], d) : bv[a][e][c];
          sum = add_rn(sum, resid(bb, d, xv[a][e][c], wsum(F, ax, ay, az)));
        }
    bc[lrow(Cl, i, j, k)] = mul_rn(sum, inv);
  }
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_mg_prolong8(MgLevelT<T> F, MgLevelT<T> Cl, const T *__restrict__ xc,
                                                        T *__restrict__ xf, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  const long long sx = (long long)F.ny * F.nz, sy = F.nz;
  FOR_LEVEL(Cl) {
    // the 3 x 3 x 3 coarse neighbourhood; beyond a wall the parent's value (axis_taps)
    T cv[3][3][3];
    const int ci[3] = {i > 0 ? i - 1 : i, i, i < Cl.nx - 1 ? i + 1 : i};
    const int cj[3] = {j > 0 ? j - 1 : j, j, j < Cl.ny - 1 ? j + 1 : j};
    const int ck[3] = {k > 0 ? k - 1 : (Cl.pz ? Cl.nz - 1 : k), k, k < Cl.nz - 1 ? k + 1 : (Cl.pz ? 0 : k)};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int e = 0; e < 3; ++e)
#pragma unroll
        for (int c = 0; c < 3; ++c) cv[a][e][c] = xc[lrow(Cl, ci[a], cj[e], ck[c])];
    const T w0 = T(0.75), w1 = T(0.25);
    const long long r0 = lrow(F, 2 * i, 2 * j, 2 * k);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        T out[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          // taps: the parent (index 1) and the neighbour on the child's side (0 or 2), in
          // k_mg_prolong's order (parent first on every axis) and weights
          const int ti[2] = {1, a ? 2 : 0}, tj[2] = {1, e ? 2 : 0}, tk[2] = {1, c ? 2 : 0};
          const T wa[2] = {w0, w1};
          T v = T(0);
#pragma unroll
          for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
              for (int t = 0; t < 2; ++t) v = fma_rn(wa[p] * wa[q] * wa[t], cv[ti[p]][tj[q]][tk[t]], v);
          out[c] = v;
        }
        T *dst = xf + r0 + a * sx + e * sy;
        T x0, x1;
        ld2(dst, x0, x1);
        st2(dst, add_rn(x0, out[0]), add_rn(x1, out[1]));
      }
  }
}

// ---- FP64 levels with an even nz (the FP64 hierarchy): one thread per pair of cells along k,
// of which one has the pass's colour, so that no lane idles.  These passes are bound by the
// FP64 pipe (one warp instruction per 64 cycles and scheduler, idle lanes included), so the
// same V-cycle is formed with few FP64 operations:
//   - a missing neighbour is a zero selected on the integer pipe, not a guarded addition;
//   - Jacobi-scaled rows (b' = b / diag): x0 from zero is b' itself, so the first pass reads
//     its colour-0 neighbours from b' and stores both colours, and later passes take
//     b' + idg S instead of (diag b' + S) idg;
//   - after the pre-smoothing the residual is zero on colour 1 and, on colour 0, just the
//     weighted sum of the colour-1 neighbours (x0 = b / diag), so the restriction reads no b;
//   - the prolongation is added on colour 0 only: the next pass overwrites colour 1.
// About 19 FP64 instructions a cell and V-cycle against 85 (and half the lanes idle) in the
// general kernels above, which the levels with an odd nz keep.  512x256x64: a V-cycle
// 1.44 -> 0.44 ms.
#define FOR_PAIRS(L)                                          \
  const int kp = blockIdx.x * blockDim.x + threadIdx.x;       \
  const int j = blockIdx.y * blockDim.y + threadIdx.y;        \
  const bool on_ = (kp < ((L).nz >> 1)) && (j < (L).ny);      \
  for (int i = blockIdx.z; on_ && i < (L).nx; i += gridDim.z)

// weighted sum of the neighbours' values (lnb: the three pair sums, then the weights)
__device__ __forceinline__ double lnb64(const MgLevelT<double> &L, const double *x, int i, int j, int k, long long r,
                                        double start) {
  const long long sx = (long long)L.ny * L.nz;
  const double xm = i > 0 ? x[r - sx] : 0.0, xp = i < L.nx - 1 ? x[r + sx] : 0.0;
  const double ym = j > 0 ? x[r - L.nz] : 0.0, yp = j < L.ny - 1 ? x[r + L.nz] : 0.0;
  const double zm = k > 0 ? x[r - 1] : (L.pz ? x[r + L.nz - 1] : 0.0);
  const double zp = k < L.nz - 1 ? x[r + 1] : (L.pz ? x[r + 1 - L.nz] : 0.0);
  return fma_rn(L.wz, zm + zp, fma_rn(L.wy, ym + yp, fma_rn(L.wx, xm + xp, start)));
}

// x = b / diag on colour 0 (from zero; unscaled rows)
__global__ void __launch_bounds__(kBlock) k_mgp_scale(MgLevelT<double> L, const double *__restrict__ b,
                                                      double *__restrict__ x, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  FOR_PAIRS(L) {
    const int k = 2 * kp + ((i + j) & 1);
    const long long r = lrow(L, i, j, k);
    x[r] = b[r] * linv(L, i, j, k);
  }
}

// one colour from the other: x = (b + S) idg, or b' + idg S for Jacobi-scaled rows (JAC);
// from_b: the other colour's values are b' and are stored too (the first pass on JAC rows)
template <bool JAC>
__global__ void __launch_bounds__(kBlock) k_mgp_colour(MgLevelT<double> L, int colour, int from_b,
                                                       const double *__restrict__ b, double *x, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  const double *nb = from_b ? b : x;
  FOR_PAIRS(L) {
    const int d = (i + j + colour) & 1, k = 2 * kp + d;
    const long long r = lrow(L, i, j, k);
    const double idg = linv(L, i, j, k);
    x[r] = JAC ? fma_rn(lnb64(L, nb, i, j, k, r, 0.0), idg, b[r]) : lnb64(L, nb, i, j, k, r, b[r]) * idg;
    if (from_b) x[r + 1 - 2 * d] = b[r + 1 - 2 * d];
  }
}

// bc = average over the children of the residual: the colour-1 neighbours of the four
// colour-0 children (every axis halves)
__global__ void __launch_bounds__(kBlock) k_mgp_restrict(MgLevelT<double> F, MgLevelT<double> Cl,
                                                         const double *__restrict__ x, double *__restrict__ bc,
                                                         const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  const long long sx = (long long)F.ny * F.nz, sy = F.nz;
  FOR_LEVEL(Cl) {
    double a = 0.0, e = 0.0, f = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // children (0,0,0), (0,1,1), (1,0,1), (1,1,0)
      const int da = q >> 1, de = q & 1, dc = da ^ de;
      const int fi = 2 * i + da, fj = 2 * j + de, fk = 2 * k + dc;
      const long long r = lrow(F, fi, fj, fk);
      const double xm = fi > 0 ? x[r - sx] : 0.0, xp = fi < F.nx - 1 ? x[r + sx] : 0.0;
      const double ym = fj > 0 ? x[r - sy] : 0.0, yp = fj < F.ny - 1 ? x[r + sy] : 0.0;
      const double zm = fk > 0 ? x[r - 1] : (F.pz ? x[r + F.nz - 1] : 0.0);
      const double zp = fk < F.nz - 1 ? x[r + 1] : (F.pz ? x[r + 1 - F.nz] : 0.0);
      a = q == 0 ? xm + xp : a + (xm + xp);
      e = q == 0 ? ym + yp : e + (ym + yp);
      f = q == 0 ? zm + zp : f + (zm + zp);
    }
    bc[lrow(Cl, i, j, k)] = wsum(F, a, e, f) * 0.125;
  }
}

// x += P xc on colour 0 (every axis halves): k_mg_prolong8's taps
__global__ void __launch_bounds__(kBlock) k_mgp_prolong(MgLevelT<double> F, MgLevelT<double> Cl,
                                                        const double *__restrict__ xc, double *__restrict__ x,
                                                        const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  FOR_LEVEL(Cl) {
    double cv[3][3][3];
    const int ci[3] = {i > 0 ? i - 1 : i, i, i < Cl.nx - 1 ? i + 1 : i};
    const int cj[3] = {j > 0 ? j - 1 : j, j, j < Cl.ny - 1 ? j + 1 : j};
    const int ck[3] = {k > 0 ? k - 1 : (Cl.pz ? Cl.nz - 1 : k), k, k < Cl.nz - 1 ? k + 1 : (Cl.pz ? 0 : k)};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int e = 0; e < 3; ++e)
#pragma unroll
        for (int c = 0; c < 3; ++c) cv[a][e][c] = xc[lrow(Cl, ci[a], cj[e], ck[c])];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int da = q >> 1, de = q & 1, dc = da ^ de;
      const long long r = lrow(F, 2 * i + da, 2 * j + de, 2 * k + dc);
      double v = x[r];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int ta = (t >> 2) & 1, te = (t >> 1) & 1, tc = t & 1;
        const double w = (ta ? 0.25 : 0.75) * (te ? 0.25 : 0.75) * (tc ? 0.25 : 0.75);
        v = fma_rn(w, cv[ta ? 2 * da : 1][te ? 2 * de : 1][tc ? 2 * dc : 1], v);
      }
      x[r] = v;
    }
  }
}

// ---- a level whose every axis halves, FP32, nz / 4 up to kMgMarchQuads: its V-cycle work in
// two marching kernels instead of six per-pass launches.  A block of nz / 4 x (mty / 2 + 2)
// threads owns a band of mty rows and two halo rows on each side (a thread: one quad along k of
// two rows, j even and j + 1) and marches along x over a segment of msx planes and two halo
// planes on each side.  The cells of one colour in a quad are a pair: the even or the odd ones,
// by the row's parity (E, O below), known at compile time since the rows are j even and odd and
// the planes are unrolled.  The x and y neighbours of one colour's pair are the other colour's
// pairs of the planes and rows beside it, its z neighbours that pair itself and the same
// shifted by one, so every colour pass is FP32x2 arithmetic on the cells of its colour only.
// A thread's own planes stay in registers (rings of three); the neighbours' rows and quads come
// from shared memory, two buffers a colour and one barrier a plane:
//   step p: colour 0 of plane p, colour 1 of plane p - 1, the last stage of plane p - 2, from
//   the neighbours' pairs of the planes that the step before wrote.
//   k_mg_down: the pre-smoothing from zero (colour 0: b / diag; colour 1 from those), the
//     residual (colour 1's from its update's own neighbour sum) and its restriction to the
//     next level's b.  The level's x is not stored: the only part of it read later, colour
//     0's, is b / diag again.
//   k_mg_up: colour 0 = b / diag + P xc, then the colour-1 and colour-0 passes of the
//     post-smoothing; x stored.
// Neighbours beyond a wall enter as zeros.  Each value is otherwise formed by the rounded
// sequence of k_mg_smooth4, k_mg_restrict8 or k_mg_prolong8 (the pair operations round each
// component as the scalar ones do), so a V-cycle gives the per-pass kernels' result (equal as
// numbers: a sum of two zeros may differ in sign).
constexpr int kMgMarchThreads = 512;
constexpr int kMgMarchQuads = 128;  // at least four row pairs a block

__device__ __forceinline__ float2 pr(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 bc2(float a) { return make_float2(a, a); }
// a product that enters a sum: scalar, since the compiler contracts a pair product that feeds a
// pair sum into one FFMA2 (results different from the per-pass kernels' rounded product)
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return pr(mul_rn(a.x, b.x), mul_rn(a.y, b.y)); }
// (scalar: the prolongation's operands are not aligned register pairs)
__device__ __forceinline__ float2 fma2s(float2 a, float2 b, float2 c) {
  return pr(fma_rn(a.x, b.x, c.x), fma_rn(a.y, b.y, c.y));
}
// wsum of two cells
__device__ __forceinline__ float2 wsum2(const MgLevel &L, float2 a, float2 e, float2 f) {
  return __ffma2_rn(bc2(L.wz), f, __ffma2_rn(bc2(L.wy), e, __fmul2_rn(bc2(L.wx), a)));
}

// 1/diag (x, y) and the diagonal (z, w) of a quad's even or odd cells, in shared memory by
// [one x neighbour or two][y neighbours, 3: a row beyond the level (1/diag 0: colour 1 is zero
// there)][z neighbour before][after][even, odd]; one entry serves all threads of a kind (as
// registers, with a branch at the first and last plane: 17 % slower on 512x256x64)
struct MarchDiag {
  float4 v[2][4][2][2][2];
};
__device__ __forceinline__ void march_diag(const MgLevel &L, MarchDiag &D) {
  for (int t = threadIdx.x; t < 64; t += blockDim.x) {
    const int odd = t & 1, zr = (t >> 1) & 1, zl = (t >> 2) & 1, cy = (t >> 3) & 3, cx = 1 + (t >> 5);
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    if (cy < 3) {
      const int c = 9 * cx + 3 * cy, c0 = odd ? 2 : 1 + zl, c1 = odd ? 1 + zr : 2;
      const float dxy = add_rn(L.wx * (float)cx, L.wy * (float)cy);  // the products are exact
      d = make_float4(L.idg[c + c0], L.idg[c + c1], add_rn(dxy, L.wz * (float)c0), add_rn(dxy, L.wz * (float)c1));
    }
    (&D.v[0][0][0][0][0])[t] = d;
  }
}

// a thread's rows and quad, and what does not change along the march
struct MarchRows {
  int q, ty, j;       // j: the even row (-2: below the level)
  bool in, band;      // the rows exist; and belong to the band
  bool zl, zr;        // the quad has a z neighbour before / after it (or across the wrap)
  int im, ip, il, ir; // threads of the rows below and above, of the quads before and after
  int d[2];           // the rows' entries of MarchDiag (even cells, one x neighbour)
  // row r's even (odd = 0) or odd cells on plane i
  __device__ __forceinline__ float4 diag(const MgLevel &L, const MarchDiag &D, int r, int odd, int i) const {
    return (&D.v[0][0][0][0][0])[d[r] + (i > 0 && i < L.nx - 1 ? 32 : 0) + odd];  // (a march has nx >= 2)
  }
};

__device__ __forceinline__ MarchRows march_rows(const MgLevel &L) {
  MarchRows R;
  const int nq = L.nz >> 2, tid = threadIdx.x, rows = blockDim.x / nq;
  R.ty = tid / nq;
  R.q = tid - R.ty * nq;
  R.j = blockIdx.y * L.mty - 2 + 2 * R.ty;
  R.in = R.j >= 0 && R.j < L.ny;  // ny is even: both rows or neither
  R.band = R.in && R.ty >= 1 && R.ty < rows - 1;
  R.zl = R.q > 0 || L.pz;
  R.zr = R.q < nq - 1 || L.pz;
  // (the outer halo rows' missing neighbours: any value, used by no row that is)
  R.im = R.ty > 0 ? tid - nq : tid;
  R.ip = R.ty < rows - 1 ? tid + nq : tid;
  R.il = R.q > 0 ? tid - 1 : tid + nq - 1;
  R.ir = R.q < nq - 1 ? tid + 1 : tid + 1 - nq;
#pragma unroll
  for (int r = 0; r < 2; ++r)
    R.d[r] = 8 * (R.in ? (R.j + r > 0) + (R.j + r < L.ny - 1) : 3) + 4 * (int)R.zl + 2 * (int)R.zr;
  return R;
}

// the pairs beside a colour's cells along z: own, the other colour's pair of the quad; nb, the
// one that lies beyond the quad (odd: the cells are the odd ones, else the even ones)
__device__ __forceinline__ float2 march_z(int odd, float2 own, float nb) {
  return odd ? __fadd2_rn(own, pr(own.y, nb)) : __fadd2_rn(pr(nb, own.x), own);
}
// that value: the last cell of the quad before or the first of the one after, zero beyond a wall
__device__ __forceinline__ float march_zn(const MarchRows &R, int odd, const float2 *s) {
  return odd ? (R.zr ? s[R.ir].x : 0.f) : (R.zl ? s[R.il].y : 0.f);
}
__device__ __forceinline__ float2 lo2(float4 v) { return pr(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return pr(v.z, v.w); }
__device__ __forceinline__ float2 neg2(float2 v) { return pr(-v.x, -v.y); }

// the march over planes p = is - 2 .. ie + 1, six at a time: the planes' parity and the places
// in the rings of three are compile-time
#define CFDGB_MARCH_PLANES(STEP)                             \
  for (int p = is - 2;;) {                                   \
    STEP(p, std::integral_constant<int, 0>{});               \
    if (++p > ie + 1) break;                                 \
    STEP(p, std::integral_constant<int, 1>{});               \
    if (++p > ie + 1) break;                                 \
    STEP(p, std::integral_constant<int, 2>{});               \
    if (++p > ie + 1) break;                                 \
    STEP(p, std::integral_constant<int, 3>{});               \
    if (++p > ie + 1) break;                                 \
    STEP(p, std::integral_constant<int, 4>{});               \
    if (++p > ie + 1) break;                                 \
    STEP(p, std::integral_constant<int, 5>{});               \
    if (++p > ie + 1) break;                                 \
    six();                                                   \
  }

template <bool BS>
__global__ void __launch_bounds__(kMgMarchThreads)
    k_mg_down(MgLevel F, MgLevel Cl, const float *__restrict__ b, float *__restrict__ bc, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  // the pairs of both rows of every thread: [buffer][row][thread]
  __shared__ float2 s0[2][2][kMgMarchThreads], s1[2][2][kMgMarchThreads];
  __shared__ MarchDiag D;
  const int tid = threadIdx.x;
  const MarchRows R = march_rows(F);
  march_diag(F, D);
  __syncthreads();
  const int is = blockIdx.x * F.msx, ie = min(F.nx, is + F.msx);
  const int sx = F.ny * F.nz, o = (R.in ? R.j : 0) * F.nz + 4 * R.q;  // 32-bit: under 2^31 cells
  auto ldb = [&](int p, int r) -> float4 {
    return R.in && p >= 0 && p < F.nx ? __ldg(reinterpret_cast<const float4 *>(b + (o + r * F.nz + p * sx)))
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  float4 bn[2][2];  // b of the next two planes
  float2 b0[3][2], b1[3][2], c0[3][2], c1[3][2], r1[3][2];  // b, x of each colour, colour 1's residual
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    bn[0][r] = ldb(is - 2, r);
    bn[1][r] = ldb(is - 1, r);
#pragma unroll
    for (int t = 0; t < 3; ++t) b0[t][r] = b1[t][r] = c0[t][r] = c1[t][r] = r1[t][r] = pr(0.f, 0.f);
  }
  float2 S = pr(0.f, 0.f);  // the restriction sums of the quad's two coarse cells
  auto step = [&](int p, auto u) {
    constexpr int U = decltype(u)::value, P = U % 3, Q = (U + 2) % 3, T = (U + 1) % 3, W = U & 1;
#pragma unroll
    for (int r = 0; r < 2; ++r) {  // plane p: b, and colour 0 from zero (zeros outside the level)
      const int par = W ^ r;
      const float4 v = bn[W][r], d = R.diag(F, D, r, par, p);
      bn[W][r] = ldb(p + 2, r);
      b0[P][r] = par ? pr(v.y, v.w) : pr(v.x, v.z);
      b1[P][r] = par ? pr(v.x, v.z) : pr(v.y, v.w);
      if (BS) {  // Jacobi-scaled rows
        b0[P][r] = mul2(b0[P][r], hi2(d));
        b1[P][r] = mul2(b1[P][r], hi2(R.diag(F, D, r, 1 - par, p)));
      }
      c0[P][r] = mul2(b0[P][r], lo2(d));
    }
    {  // plane p - 1: colour 1 from colour 0, and its residual from the same neighbour sum
      const int i = p - 1;
      if (i >= 0 && i < F.nx) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int odd = W ^ r;  // the row's colour-0 cells on plane i are the other ones
          const float2 a = __fadd2_rn(c0[T][r], c0[P][r]);
          const float2 e = __fadd2_rn(r ? c0[Q][0] : s0[1 - W][1][R.im], r ? s0[1 - W][0][R.ip] : c0[Q][1]);
          const float2 w = wsum2(F, a, e, march_z(odd, c0[Q][r], march_zn(R, odd, s0[1 - W][r])));
          const float4 d = R.diag(F, D, r, odd, i);
          c1[Q][r] = mul2(__fadd2_rn(b1[Q][r], w), lo2(d));
          r1[Q][r] = __fadd2_rn(__ffma2_rn(neg2(hi2(d)), c1[Q][r], b1[Q][r]), w);
        }
      } else {
        c1[Q][0] = c1[Q][1] = pr(0.f, 0.f);
      }
    }
    {  // plane p - 2: colour 0's residual, and the restriction (k_mg_restrict8's sums)
      const int i = p - 2;
      if (i >= is) {
        if (!W) S = pr(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int odd = W ^ r;
          const float2 a = __fadd2_rn(c1[P][r], c1[Q][r]);
          const float2 e = __fadd2_rn(r ? c1[T][0] : s1[W][1][R.im], r ? s1[W][0][R.ip] : c1[T][1]);
          const float2 w = wsum2(F, a, e, march_z(odd, c1[T][r], march_zn(R, odd, s1[W][r])));
          const float2 d = hi2(R.diag(F, D, r, odd, i));
          const float2 r0 = __fadd2_rn(__ffma2_rn(neg2(d), c0[T][r], b0[T][r]), w);
          S = __fadd2_rn(__fadd2_rn(S, odd ? r1[T][r] : r0), odd ? r0 : r1[T][r]);
        }
        if (W && R.band) {
          const float inv = 1.f / 8.f;
          *reinterpret_cast<float2 *>(bc + lrow(Cl, i >> 1, R.j >> 1, 2 * R.q)) =
              make_float2(mul_rn(S.x, inv), mul_rn(S.y, inv));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      s0[W][r][tid] = c0[P][r];
      s1[1 - W][r][tid] = c1[Q][r];
    }
    __syncthreads();
  };
  auto six = [] {};
  CFDGB_MARCH_PLANES(step)
}

template <bool BS>
__global__ void __launch_bounds__(kMgMarchThreads)
    k_mg_up(MgLevel F, MgLevel Cl, const float *__restrict__ b, const float *__restrict__ xc, float *__restrict__ x,
            const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  __shared__ float2 s0[2][2][kMgMarchThreads], s1[2][2][kMgMarchThreads];
  __shared__ float2 sc_[kMgMarchThreads + 2 * kMgMarchQuads];  // a coarse plane: the rows' parents, one row more on each side
  __shared__ MarchDiag D;
  const int tid = threadIdx.x, nq = F.nz >> 2;
  const MarchRows R = march_rows(F);
  march_diag(F, D);
  const int is = blockIdx.x * F.msx, ie = min(F.nx, is + F.msx);
  const int sx = F.ny * F.nz, o = (R.in ? R.j : 0) * F.nz + 4 * R.q;  // 32-bit: under 2^31 cells
  auto ldb = [&](int p, int r) -> float4 {
    return R.in && p >= 0 && p < F.nx ? __ldg(reinterpret_cast<const float4 *>(b + (o + r * F.nz + p * sx)))
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  // the parents of the thread's rows (a coarse row, clamped to the level) and, in the first and
  // last rows of threads, the coarse row before and after
  const int pj = R.j >> 1, csx = Cl.ny * Cl.nz, c2 = 2 * R.q;
  const bool first = R.ty == 0, last = tid + nq >= (int)blockDim.x;
  const int co = min(max(pj, 0), Cl.ny - 1) * Cl.nz + c2;
  const int cx = min(max(first ? pj - 1 : pj + 1, 0), Cl.ny - 1) * Cl.nz + c2;
  float2 n0, n1 = pr(0.f, 0.f);  // the next coarse plane on its way
  auto ldc = [&](int m) {
    const int t = min(max(m, 0), Cl.nx - 1) * csx;
    n0 = __ldg(reinterpret_cast<const float2 *>(xc + (t + co)));
    if (first || last) n1 = __ldg(reinterpret_cast<const float2 *>(xc + (t + cx)));
  };
  auto putc = [&] {
    sc_[tid + nq] = n0;
    if (first) sc_[tid] = n1;
    if (last) sc_[tid + 2 * nq] = n1;
  };
  // a coarse plane's values for the quad: rows pj, pj - 1, pj + 1 x coarse z 2q - 1 .. 2q + 2, the
  // ends the parent beyond a wall or wrapped (k_mg_prolong8's taps)
  const float *const cf = reinterpret_cast<const float *>(sc_);
  const int kl = R.zl ? 2 * R.il + 1 : 2 * tid, kr = R.zr ? 2 * R.ir : 2 * tid + 1;
  auto getc = [&](float (&v)[3][4]) {
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const int d = t == 0 ? nq : (t == 1 ? 0 : 2 * nq);
      const float2 c = sc_[tid + d];
      v[t][0] = cf[kl + 2 * d];
      v[t][1] = c.x;
      v[t][2] = c.y;
      v[t][3] = cf[kr + 2 * d];
    }
  };
  // (is - 2 is even: the march starts on a first child.)  cv[0], cv[1]: the coarse planes m - 1
  // and m of the parent plane m = p / 2, m + 1 replacing m - 1 on the second child
  const int m0 = (is - 2) >> 1;
  float cv[2][3][4];
  ldc(m0 - 1);
  putc();
  __syncthreads();
  getc(cv[0]);
  ldc(m0);
  __syncthreads();
  putc();
  __syncthreads();
  getc(cv[1]);
  ldc(m0 + 1);
  __syncthreads();
  float4 bn[2][2];  // b of the next two planes
  float2 b0[3][2], b1[3][2], c0[3][2], c1[3][2];  // b and x of each colour
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    bn[0][r] = ldb(is - 2, r);
    bn[1][r] = ldb(is - 1, r);
#pragma unroll
    for (int t = 0; t < 3; ++t) b0[t][r] = b1[t][r] = c0[t][r] = c1[t][r] = pr(0.f, 0.f);
  }
  auto step = [&](int p, auto u) {
    constexpr int U = decltype(u)::value, P = U % 3, Q = (U + 2) % 3, T = (U + 1) % 3, W = U & 1;
    constexpr int M = 1 - (U / 2) % 2;  // cv[M]: the parent plane
    if (W) {
      getc(cv[1 - M]);
    } else {
      putc();  // plane m + 1, read on the second child
      ldc((p >> 1) + 2);
    }
    const bool plane = p >= 0 && p < F.nx;
#pragma unroll
    for (int r = 0; r < 2; ++r) {  // plane p: colour 0 = b / diag + P xc (k_mg_prolong8: parent first on every axis)
      const int par = W ^ r;
      const float4 v = bn[W][r], d = R.diag(F, D, r, par, p);
      bn[W][r] = ldb(p + 2, r);
      b0[P][r] = par ? pr(v.y, v.w) : pr(v.x, v.z);
      b1[P][r] = par ? pr(v.x, v.z) : pr(v.y, v.w);
      if (BS) {  // Jacobi-scaled rows
        b0[P][r] = mul2(b0[P][r], hi2(d));
        b1[P][r] = mul2(b1[P][r], hi2(R.diag(F, D, r, 1 - par, p)));
      }
      const float wt[2] = {0.75f, 0.25f};
      float2 t = pr(0.f, 0.f);
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float *c = cv[a ? 1 - M : M][e ? 1 + r : 0];
          const float2 w0 = bc2(wt[a] * wt[e] * wt[0]), w1 = bc2(wt[a] * wt[e] * wt[1]);
          t = a + e == 0 ? mul2(w0, pr(c[1], c[2])) : fma2s(w0, pr(c[1], c[2]), t);
          t = fma2s(w1, par ? pr(c[2], c[3]) : pr(c[0], c[1]), t);
        }
      t = __fadd2_rn(mul2(b0[P][r], lo2(d)), t);
      c0[P][r] = R.in && plane ? t : pr(0.f, 0.f);
    }
    {  // plane p - 1: colour 1 of the post-smoothing
      const int i = p - 1;
      if (i >= 0 && i < F.nx) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int odd = W ^ r;
          const float2 a = __fadd2_rn(c0[T][r], c0[P][r]);
          const float2 e = __fadd2_rn(r ? c0[Q][0] : s0[1 - W][1][R.im], r ? s0[1 - W][0][R.ip] : c0[Q][1]);
          const float2 w = wsum2(F, a, e, march_z(odd, c0[Q][r], march_zn(R, odd, s0[1 - W][r])));
          c1[Q][r] = mul2(__fadd2_rn(b1[Q][r], w), lo2(R.diag(F, D, r, odd, i)));
        }
      } else {
        c1[Q][0] = c1[Q][1] = pr(0.f, 0.f);
      }
    }
    {  // plane p - 2: colour 0, stored
      const int i = p - 2;
      if (i >= is) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int odd = W ^ r;
          const float2 a = __fadd2_rn(c1[P][r], c1[Q][r]);
          const float2 e = __fadd2_rn(r ? c1[T][0] : s1[W][1][R.im], r ? s1[W][0][R.ip] : c1[T][1]);
          const float2 w = wsum2(F, a, e, march_z(odd, c1[T][r], march_zn(R, odd, s1[W][r])));
          const float2 v = mul2(__fadd2_rn(b0[T][r], w), lo2(R.diag(F, D, r, odd, i)));
          const float2 ev = odd ? c1[T][r] : v, ov = odd ? v : c1[T][r];
          if (R.band)
            *reinterpret_cast<float4 *>(x + (o + r * F.nz + i * sx)) = make_float4(ev.x, ov.x, ev.y, ov.y);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      s0[W][r][tid] = c0[P][r];
      s1[1 - W][r][tid] = c1[Q][r];
    }
    __syncthreads();
  };
  auto six = [&] {  // three parents: the two coarse planes change places
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float v = cv[0][t][c];
        cv[0][t][c] = cv[1][t][c];
        cv[1][t][c] = v;
      }
  };
  CFDGB_MARCH_PLANES(step)
}
#undef CFDGB_MARCH_PLANES

// coarsest level: x = 0, then `sweeps` red-black sweeps in shared memory, one block
// x = M b on the coarsest level with the precomputed pseudo-inverse M (n x n, by columns, so that
// the threads of neighbouring cells read neighbouring elements): one dot product of length n per
// cell, its elements fetched sixteen at a time (the block's shared copies of b, x)
template <typename T>
__device__ __forceinline__ T dense_row(int n, const T *M, const T *bs, int q) {
  T v = T(0);
  int c = 0;
  for (; c + 16 <= n; c += 16) {
    T m[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) m[e] = M[(c + e) * n + q];
#pragma unroll
    for (int e = 0; e < 16; ++e) v = fma_rn(m[e], bs[c + e], v);
  }
  for (; c < n; ++c) v = fma_rn(M[c * n + q], bs[c], v);
  return v;
}
template <typename T>
__device__ void blk_dense(int n, const T *__restrict__ M, const T *bs, T *xs) {
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    xs[q] = dense_row(n, M, bs, q);
  }
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(1024) k_mg_coarse(MgLevelT<T> L, int sweeps, const T *__restrict__ M, int bscale,
                                                    const T *__restrict__ b, T *__restrict__ x, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smraw[];
  T *sm = reinterpret_cast<T *>(smraw);
  const int n = L.nx * L.ny * L.nz;
  T *xs = sm, *bs = sm + n;
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    const int k = q % L.nz, t = q / L.nz, j = t % L.ny, i = t / L.ny;
    T bb = b[q];
    if (bscale) bb *= ldiag(L, i, j, k);
    bs[q] = bb;
    xs[q] = T(0);
  }
  __syncthreads();
  if (M) {
    blk_dense(n, M, bs, xs);
    sweeps = 0;
  }
  for (int s = 0; s < sweeps; ++s)
    for (int colour = 0; colour < 2; ++colour) {
      for (int q = threadIdx.x; q < n; q += blockDim.x) {
        const int k = q % L.nz, t = q / L.nz, j = t % L.ny, i = t / L.ny;
        if (((i + j + k) & 1) != colour) continue;
        xs[q] = (bs[q] + lnb(L, xs, i, j, k, q)) * linv(L, i, j, k);
      }
      __syncthreads();
    }
  for (int q = threadIdx.x; q < n; q += blockDim.x) x[q] = xs[q];
}

// ---- the small levels in one block: levels t..nlev-1 together hold at most
// kMgTailBytes / (2 sizeof(T)) cells, x and b of each in shared memory; the same smoothing,
// transfers and coarsest solve as the per-level kernels (same arithmetic, same order), a
// barrier between phases where the per-level path has a launch ----
// 48 KB: one block working on more cells per barrier (a 16K-cell level, 192 KB) ran slower
// than the same level's launched kernels (measured on 512x256x64)
constexpr int kMgTailBytes = 48 * 1024;
// FP64: 1024 cells.  One multiprocessor's FP64 pipe (2 lanes a clock) takes longer for a level of
// 2048 cells than that level's launched kernels: runs on 512x256x64 60.1 -> 59.2 ms, on
// 256x128x32 12.1 -> 11.1 ms against 3072 cells (48 KB); 128 cells 59.3 and 11.3 ms
template <typename T>
constexpr int tail_cells_max() {
  return sizeof(T) == sizeof(double) ? 1024 : kMgTailBytes / (2 * (int)sizeof(T));
}

// Unsigned division by an invariant d >= 1 (Granlund and Montgomery, "Division by invariant
// integers using multiplication", PLDI 1994, the round-up method): with l = ceil(log2 d) and
// m = floor(2^32 (2^l - d) / d) + 1, n / d = (t + ((n - t) >> 1)) >> (l - 1), t = mulhi(m, n),
// for every 32-bit n (d = 1: l = 0 and the quotient is n).
static inline void div_magic(unsigned d, unsigned *m, int *l) {
  int ll = 0;
  while ((1ull << ll) < d) ++ll;
  *l = ll;
  *m = (unsigned)((((1ull << ll) - d) << 32) / d + 1);
}
__device__ __forceinline__ unsigned udiv_inv(unsigned n, unsigned m, int l) {
  if (l == 0) return n;
  const unsigned t = __umulhi(m, n);
  return (t + ((n - t) >> 1)) >> (l - 1);
}

template <typename T>
__device__ __forceinline__ void cell_ijk(const MgLevelT<T> &L, int q, int &i, int &j, int &k) {
  const unsigned t = udiv_inv((unsigned)q, L.dz_m, L.dz_l), u = udiv_inv(t, L.dy_m, L.dy_l);
  k = q - (int)t * L.nz;
  j = (int)t - (int)u * L.ny;
  i = (int)u;
}

template <typename T>
__device__ void blk_smooth(const MgLevelT<T> &L, int colour, int zero, const T *b, T *x) {
  const int n = L.nx * L.ny * L.nz;
  if constexpr (sizeof(T) == sizeof(double)) {
    if (L.nz % 2 == 0) {  // k_mgp_scale, k_mgp_colour
      const int half = L.nz / 2, np = n / 2;
      for (int p = threadIdx.x; p < np; p += blockDim.x) {
        const unsigned r = udiv_inv((unsigned)p, L.dh_m, L.dh_l), ii = udiv_inv(r, L.dy_m, L.dy_l);
        const int i = (int)ii, j = (int)r - i * L.ny, d = (i + j + colour) & 1;
        const int k = 2 * (p - (int)r * half) + d, q = (int)r * L.nz + k;
        x[q] = (zero ? b[q] : lnb64(L, x, i, j, k, q, b[q])) * linv(L, i, j, k);
      }
      __syncthreads();
      return;
    }
  }
  if (L.nz % 2 == 0) {
    // the cells of a row pair up along k, one of each colour: a thread per pair updates the
    // one of the colour (and, from zero, clears the other)
    const int half = L.nz / 2, np = n / 2;
    for (int p = threadIdx.x; p < np; p += blockDim.x) {
      const unsigned r = udiv_inv((unsigned)p, L.dh_m, L.dh_l), ii = udiv_inv(r, L.dy_m, L.dy_l);
      const int i = (int)ii, j = (int)r - i * L.ny, d = (i + j + colour) & 1;
      const int k = 2 * (p - (int)r * half) + d, q = (int)r * L.nz + k;
      if (zero) x[q + 1 - 2 * d] = T(0);
      const T num = zero ? b[q] : b[q] + lnb(L, x, i, j, k, q);
      x[q] = num * linv(L, i, j, k);
    }
    __syncthreads();
    return;
  }
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    int i, j, k;
    cell_ijk(L, q, i, j, k);
    if (((i + j + k) & 1) != colour) {
      if (zero) x[q] = T(0);
      continue;
    }
    const T num = zero ? b[q] : b[q] + lnb(L, x, i, j, k, q);
    x[q] = num * linv(L, i, j, k);
  }
  __syncthreads();
}

template <typename T>
__device__ void blk_restrict(const MgLevelT<T> &F, const MgLevelT<T> &Cl, const T *bf, const T *xf, T *bc) {
  const T inv = T(1) / (T)(F.fx * F.fy * F.fz);
  const int n = Cl.nx * Cl.ny * Cl.nz;
  const bool pairs = sizeof(T) == sizeof(double) && F.nz % 2 == 0;  // zero residual on colour 1 (k_mgp_restrict)
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    int i, j, k;
    cell_ijk(Cl, q, i, j, k);
    T sum = T(0);
    if constexpr (sizeof(T) == sizeof(double)) {
      if (pairs) {
        for (int a = 0; a < F.fx; ++a)
          for (int e = 0; e < F.fy; ++e)
            for (int c = 0; c < F.fz; ++c) {
              const int fi = i * F.fx + a, fj = j * F.fy + e, fk = k * F.fz + c;
              if (!((fi + fj + fk) & 1)) sum = lnb64(F, xf, fi, fj, fk, lrow(F, fi, fj, fk), sum);
            }
        bc[q] = sum * inv;
        continue;
      }
    }
    for (int a = 0; a < F.fx; ++a)
      for (int e = 0; e < F.fy; ++e)
        for (int c = 0; c < F.fz; ++c) {
          const int fi = i * F.fx + a, fj = j * F.fy + e, fk = k * F.fz + c;
          const long long r = lrow(F, fi, fj, fk);
          const T d = ldiag(F, fi, fj, fk);
          sum += bf[r] - d * xf[r] + lnb(F, xf, fi, fj, fk, r);
        }
    bc[q] = sum * inv;
  }
  __syncthreads();
}

template <typename T>
__device__ void blk_prolong(const MgLevelT<T> &F, const MgLevelT<T> &Cl, const T *xc, T *xf) {
  const int n = F.nx * F.ny * F.nz;
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    int i, j, k;
    cell_ijk(F, q, i, j, k);
    if (sizeof(T) == sizeof(double) && F.nz % 2 == 0 && ((i + j + k) & 1)) continue;  // overwritten next
    xf[q] += prolong_at(F, Cl, xc, i, j, k);
  }
  __syncthreads();
}

// x_t = V-cycle of levels t..nlev-1 on b_t (both in global memory, level t >= 1)
template <typename T>
__global__ void __launch_bounds__(1024) k_mg_tail(MgPlanT<T> mg, int t, const SolverScal *sc) {
  pdl_wait();
  if (sc->done) return;
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smraw[];
  T *sm = reinterpret_cast<T *>(smraw);
  const int n = mg.nlev;
  T *xs[kMgMaxLevels], *bs[kMgMaxLevels];
  int off = 0;
  for (int l = t; l < n; ++l) {
    const int c = mg.lev[l].nx * mg.lev[l].ny * mg.lev[l].nz;
    xs[l] = sm + off;
    bs[l] = sm + off + c;
    off += 2 * c;
  }
  const int nt = mg.lev[t].nx * mg.lev[t].ny * mg.lev[t].nz;
  for (int q = threadIdx.x; q < nt; q += blockDim.x) bs[t][q] = mg.lev[t].b[q];
  __syncthreads();
  for (int l = t; l + 1 < n; ++l) {
    blk_smooth(mg.lev[l], 0, 1, bs[l], xs[l]);
    blk_smooth(mg.lev[l], 1, 0, bs[l], xs[l]);
    blk_restrict(mg.lev[l], mg.lev[l + 1], bs[l], xs[l], bs[l + 1]);
  }
  {  // coarsest: the dense pseudo-inverse, or x = 0 and red-black sweeps (k_mg_coarse)
    const MgLevelT<T> &C = mg.lev[n - 1];
    const int nc = C.nx * C.ny * C.nz;
    if (mg.cinv) {
      blk_dense(nc, mg.cinv, bs[n - 1], xs[n - 1]);
    } else {
      for (int q = threadIdx.x; q < nc; q += blockDim.x) xs[n - 1][q] = T(0);
      __syncthreads();
      for (int s = 0; s < mg.coarse_sweeps; ++s) {
        blk_smooth(C, 0, 0, bs[n - 1], xs[n - 1]);
        blk_smooth(C, 1, 0, bs[n - 1], xs[n - 1]);
      }
    }
  }
  for (int l = n - 2; l >= t; --l) {
    blk_prolong(mg.lev[l], mg.lev[l + 1], xs[l + 1], xs[l]);
    blk_smooth(mg.lev[l], 1, 0, bs[l], xs[l]);
    blk_smooth(mg.lev[l], 0, 0, bs[l], xs[l]);
  }
  for (int q = threadIdx.x; q < nt; q += blockDim.x) mg.lev[t].x[q] = xs[t][q];
}

// The same tail for FP32 with a dense coarsest solve, built for latency: a phase of a small level
// has a few operations a cell, so index arithmetic, serial loads and instruction fetches were
// most of its time (512x256x64: a V-cycle 74 -> 62 us; 256x128x32: 43 -> 32; 120x40x12, with a
// coarsest level of 225 cells: 37 -> 25).
//   - A thread owns a pair of neighbours along an axis with an even extent (one cell of each
//     colour; every level but the coarsest halves one).  The pairs' addresses come from a table
//     made with the plan (mg_tail_table), copied to shared memory, as the coarsest level's
//     inverse is, before the kernel waits for the one before it.
//   - x is stored with a layer of ghost cells: zeros beyond walls, copies across a periodic z, so
//     a neighbour sum is six unconditional loads.
//   - The residuals go to a scratch copy of the level, one thread a pair, and the next level's
//     threads add up their cells' children (k_mg_tail: eight residuals, one after the other, a
//     thread).
//   - The prolongation forms colour 0 only: the pass that follows overwrites colour 1.
// Every value is formed by k_mg_tail's rounded sequence (lnb's sum as the compiler contracts it).
constexpr int kTailSlots = 3;             // pairs a thread
constexpr int kTailShared = 224 * 1024;  // bytes
constexpr int kTailDiag = 28;             // entries of a level's table of diagonals (27, padded)
static_assert(kTailSlots * 1024 * 2 >= tail_cells_max<float>(), "a thread's pairs");

__host__ __device__ __forceinline__ int tail_padded(const MgLevel &L) { return (L.nx + 2) * (L.ny + 2) * (L.nz + 2); }
__host__ __device__ __forceinline__ int tail_cells(const MgLevel &L) { return L.nx * L.ny * L.nz; }

// shared memory in words: [pairs and coarsest cells][1/diag and diag][x, padded][b][the coarsest level's
// b][scratch][inverse, the columns that fit]; the first two as in the table in global memory
struct TailLayout {
  int tab, x, b, d, s, m, cols, words;
};
static TailLayout tail_layout(const MgPlan &mg) {
  TailLayout o;
  int pairs = 0, px = 0;
  for (int l = mg.tail; l < mg.nlev; ++l) {
    px += tail_padded(mg.lev[l]);
    if (l < mg.nlev - 1) pairs += tail_cells(mg.lev[l]) / 2;
  }
  const int nc = tail_cells(mg.lev[mg.nlev - 1]), all = kTailShared / 4;
  o.tab = 4 * (pairs + nc);
  o.x = o.tab + 2 * kTailDiag * (mg.nlev - 1 - mg.tail);
  o.b = o.x + ((px + 1) & ~1);
  o.d = (o.b + 2 * pairs + 3) & ~3;
  o.s = o.d + kMgDenseCells;
  o.m = (o.s + tail_padded(mg.lev[mg.tail]) + 3) & ~3;
  o.cols = o.m >= all ? 0 : (all - o.m) / nc;
  if (o.cols >= nc) o.cols = nc;
  o.words = o.m + o.cols * nc;
  return o;
}

__device__ __forceinline__ void tail_put(const MgLevel &L, float *X, int a, int wrap, float v) {
  X[a] = v;
  if (wrap) X[a + (wrap == 1 ? L.nz : -L.nz)] = v;
}
__device__ __forceinline__ float tail_nb(const MgLevel &L, const float *X, int a) {
  const int PZ = L.nz + 2, PX = (L.ny + 2) * PZ;
  const float x = add_rn(X[a - PX], X[a + PX]), y = add_rn(X[a - PZ], X[a + PZ]), z = add_rn(X[a - 1], X[a + 1]);
  return fma_rn(L.wz, z, fma_rn(L.wx, x, mul_rn(L.wy, y)));
}
// the average of the residuals of a cell's children (k_mg_restrict's order), the first at s
__device__ __forceinline__ float tail_children(const MgLevel &F, const float *s) {
  const int PZ = F.nz + 2, PX = (F.ny + 2) * PZ;
  float v = 0.f;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (a < F.fx && e < F.fy && c < F.fz) v = add_rn(v, s[a * PX + e * PZ + c]);
  return mul_rn(v, (F.fx == 2 ? 0.5f : 1.f) * (F.fy == 2 ? 0.5f : 1.f) * (F.fz == 2 ? 0.5f : 1.f));
}

// A pair's entry (int4): x: padded addresses of the cells of colour 0 and 1 (16 bits each); y: their
// rows of the diagonal table (5 bits each), where a copy across the periodic wrap goes (2 bits
// each: 1 after, 2 before), and colour 0's side taps along x, y, z (2 bits each: 1 after, 2
// before, 0 the parent itself); z: both cells' rows of the level (the first level) or their first
// children's addresses; w: the address of colour 0's parent.  The coarsest level's cells: x: padded
// address, y: the copy across the wrap, z: the first child's address.
__device__ __forceinline__ int lo16(int v) { return v & 0xffff; }
__device__ __forceinline__ int hi16(int v) { return (int)((unsigned)v >> 16); }

__global__ void __launch_bounds__(1024) k_mg_tail32(MgPlan mg, TailLayout o, const SolverScal *sc) {
  extern __shared__ __align__(16) float tsm[];
  const int tid = threadIdx.x, n = mg.nlev, t = mg.tail;
  const MgLevel &C = mg.lev[n - 1];
  const int nc = tail_cells(C);
  const int4 *P = reinterpret_cast<const int4 *>(tsm);
  const float2 *tb = reinterpret_cast<const float2 *>(tsm + o.tab);
  float *X = tsm + o.x, *B = tsm + o.b;
  float *const S = tsm + o.s, *const D = tsm + o.d;
  {  // constants of the context: no need to wait for the kernel before
    const unsigned d = (unsigned)__cvta_generic_to_shared(tsm);
    for (int q = tid; q < o.x / 4; q += 1024)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d + 16 * q), "l"(mg.ttab + q) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int nm = o.cols * nc, n4 = nm & ~3;
    for (int q = 4 * tid; q < n4; q += 4096)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d + 4 * (o.m + q)), "l"(mg.cinv + q) : "memory");
    if (tid < nm - n4) tsm[o.m + n4 + tid] = mg.cinv[n4 + tid];
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int q = o.x + tid; q < o.b; q += 1024) tsm[q] = 0.f;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
  }
  pdl_wait();
  if (sc->done) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  pdl_trigger();
  for (int l = t; l < n - 1; ++l) {
    const MgLevel &L = mg.lev[l];
    const int np = tail_cells(L) / 2;
    int4 s[kTailSlots];
    float b[kTailSlots][2], x0[kTailSlots], r1[kTailSlots];
#pragma unroll
    for (int u = 0; u < kTailSlots; ++u) {
      const int p = tid + 1024 * u;
      if (p >= np) break;
      s[u] = P[p];
      if (l == t) {
        b[u][0] = L.b[lo16(s[u].z)];
        b[u][1] = L.b[hi16(s[u].z)];
      } else {
        b[u][0] = tail_children(mg.lev[l - 1], S + lo16(s[u].z));
        b[u][1] = tail_children(mg.lev[l - 1], S + hi16(s[u].z));
      }
      *reinterpret_cast<float2 *>(B + 2 * p) = make_float2(b[u][0], b[u][1]);
      x0[u] = mul_rn(b[u][0], tb[s[u].y & 31].x);
      tail_put(L, X, lo16(s[u].x), (s[u].y >> 10) & 3, x0[u]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTailSlots; ++u) {
      if (tid + 1024 * u >= np) break;
      const float2 d = tb[(s[u].y >> 5) & 31];
      const float w = tail_nb(L, X, hi16(s[u].x)), x1 = mul_rn(add_rn(b[u][1], w), d.x);
      r1[u] = resid(b[u][1], d.y, x1, w);
      tail_put(L, X, hi16(s[u].x), (s[u].y >> 12) & 3, x1);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTailSlots; ++u) {
      if (tid + 1024 * u >= np) break;
      const int a = lo16(s[u].x);
      S[a] = resid(b[u][0], tb[s[u].y & 31].y, x0[u], tail_nb(L, X, a));
      S[hi16(s[u].x)] = r1[u];
    }
    __syncthreads();
    X += tail_padded(L);
    B += 2 * np;
    P += np;
    tb += kTailDiag;
  }
  {  // coarsest: the dense pseudo-inverse
    const int4 s = tid < nc ? P[tid] : make_int4(0, 0, 0, 0);
    if (tid < nc) D[tid] = tail_children(mg.lev[n - 2], S + s.z);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (tid < nc) {
      // dense_row's sum; the first columns that did not fit are on their way meanwhile
      float v = 0.f, g[16];
      if (o.cols < nc) {
#pragma unroll
        for (int e = 0; e < 16; ++e) g[e] = o.cols + e < nc ? mg.cinv[(o.cols + e) * nc + tid] : 0.f;
      }
      const float *M = tsm + o.m + tid;
      int c = 0;
      for (; c + 16 <= o.cols; c += 16, M += 16 * nc) {
        float m[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) m[e] = M[e * nc];
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
          const float4 b = *reinterpret_cast<const float4 *>(D + c + e);
          v = fma_rn(m[e + 3], b.w, fma_rn(m[e + 2], b.z, fma_rn(m[e + 1], b.y, fma_rn(m[e], b.x, v))));
        }
      }
      for (; c < o.cols; ++c, M += nc) v = fma_rn(*M, D[c], v);
      if (o.cols < nc) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (o.cols + e < nc) v = fma_rn(g[e], D[o.cols + e], v);
        for (c = o.cols + 16; c < nc; ++c) v = fma_rn(mg.cinv[c * nc + tid], D[c], v);
      }
      tail_put(C, X, s.x, s.y, v);
    }
    __syncthreads();
  }
  for (int l = n - 2; l >= t; --l) {
    const MgLevel &L = mg.lev[l], &Cl = mg.lev[l + 1];
    const float *const Xc = X;
    const int np = tail_cells(L) / 2, QZ = Cl.nz + 2, QX = (Cl.ny + 2) * QZ;
    X -= tail_padded(L);
    B -= 2 * np;
    P -= np;
    tb -= kTailDiag;
    const float wi[2] = {L.fx == 2 ? 0.75f : 1.f, L.fx == 2 ? 0.25f : 0.f};
    const float wj[2] = {L.fy == 2 ? 0.75f : 1.f, L.fy == 2 ? 0.25f : 0.f};
    const float wk[2] = {L.fz == 2 ? 0.75f : 1.f, L.fz == 2 ? 0.25f : 0.f};
    int4 s[kTailSlots];
    float b[kTailSlots][2], x1[kTailSlots];
#pragma unroll
    for (int u = 0; u < kTailSlots; ++u) {  // colour 0 += P xc (prolong_at's taps in their order)
      const int p = tid + 1024 * u;
      if (p >= np) break;
      s[u] = P[p];
      const float2 v = *reinterpret_cast<const float2 *>(B + 2 * p);
      b[u][0] = v.x;
      b[u][1] = v.y;
      auto side = [&](int sh, int d) {
        const int c = (s[u].y >> sh) & 3;
        return c == 0 ? 0 : (c == 1 ? d : -d);
      };
      const int ox = side(14, QX), oy = side(16, QZ), oz = side(18, 1);
      float w = 0.f;
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int c = 0; c < 2; ++c)  // (a weight of zero adds zero times the parent)
            w = fma_rn(wi[a] * wj[e] * wk[c], Xc[s[u].w + (a ? ox : 0) + (e ? oy : 0) + (c ? oz : 0)], w);
      const int a0 = lo16(s[u].x);
      tail_put(L, X, a0, (s[u].y >> 10) & 3, add_rn(X[a0], w));
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTailSlots; ++u) {
      if (tid + 1024 * u >= np) break;
      x1[u] = mul_rn(add_rn(b[u][1], tail_nb(L, X, hi16(s[u].x))), tb[(s[u].y >> 5) & 31].x);
      tail_put(L, X, hi16(s[u].x), (s[u].y >> 12) & 3, x1[u]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTailSlots; ++u) {
      if (tid + 1024 * u >= np) break;
      const int a = lo16(s[u].x);
      const float v = mul_rn(add_rn(b[u][0], tail_nb(L, X, a)), tb[s[u].y & 31].x);
      if (l > t) {
        tail_put(L, X, a, (s[u].y >> 10) & 3, v);
      } else {
        L.x[lo16(s[u].z)] = v;
        L.x[hi16(s[u].z)] = x1[u];
      }
    }
    if (l > t) __syncthreads();
  }
}

// The pairs' entries of k_mg_tail32 for levels tail..nlev-2, the coarsest level's cells and the
// diagonals; empty:
// it cannot run this hierarchy (no tail of two levels, a coarsest level without a dense inverse,
// padded levels beyond the block's shared memory)
std::vector<int4> mg_tail_table(const MgPlan &mg) {
  std::vector<int4> tab;
  const int n = mg.nlev, nc = tail_cells(mg.lev[n - 1]);
  if (mg.tail >= n - 1 || nc > kMgDenseCells || 4ll * tail_layout(mg).m > kTailShared) return tab;
  auto addr = [](const MgLevel &L, int i, int j, int k) { return ((i + 1) * (L.ny + 2) + j + 1) * (L.nz + 2) + k + 1; };
  auto wrap = [](const MgLevel &L, int k) { return L.pz && L.nz > 1 ? (k == 0 ? 1 : (k == L.nz - 1 ? 2 : 0)) : 0; };
  auto side = [](int i, int f, int m, bool per) {
    const int d = (i & 1) ? 1 : -1, q = (i >> 1) + d;
    return f == 1 || ((q < 0 || q >= m) && !(per && m > 1)) ? 0 : (d > 0 ? 1 : 2);  // periodic: the ghost holds it
  };
  auto ends = [](int i, int m) { return (i > 0) + (i < m - 1); };
  for (int l = mg.tail; l < n; ++l) {
    const MgLevel &L = mg.lev[l], &F = mg.lev[l - 1];
    auto below = [&](int i, int j, int k) {  // the row of the level, or the first child's address
      return l == mg.tail ? (i * L.ny + j) * L.nz + k : addr(F, F.fx * i, F.fy * j, F.fz * k);
    };
    const bool coarsest = l == n - 1;
    const int di = !coarsest && L.nz % 2 && L.ny % 2, dk = !coarsest && L.nz % 2 == 0, dj = !coarsest && !di && !dk;
    for (int i = 0; i < L.nx; i += 1 + di)
      for (int j = 0; j < L.ny; j += 1 + dj)
        for (int k = 0; k < L.nz; k += 1 + dk) {
          if (coarsest) {
            tab.push_back(make_int4(addr(L, i, j, k), wrap(L, k), below(i, j, k), 0));
            continue;
          }
          int q[2][3] = {{i, j, k}, {i + di, j + dj, k + dk}};  // by colour
          if ((i + j + k) & 1) std::swap(q[0], q[1]);
          int4 e = make_int4(0, 0, 0, 0);
          for (int c = 0; c < 2; ++c) {
            const int *v = q[c];
            const int z = L.pz ? (L.nz > 1 ? 2 : 0) : ends(v[2], L.nz);
            e.x |= (int)((unsigned)addr(L, v[0], v[1], v[2]) << (16 * c));
            e.y |= (9 * ends(v[0], L.nx) + 3 * ends(v[1], L.ny) + z) << (5 * c) | wrap(L, v[2]) << (10 + 2 * c);
            e.z |= (int)((unsigned)below(v[0], v[1], v[2]) << (16 * c));
          }
          const MgLevel &Cl = mg.lev[l + 1];
          const int *v = q[0];
          e.y |= side(v[0], L.fx, Cl.nx, false) << 14 | side(v[1], L.fy, Cl.ny, false) << 16 |
                 side(v[2], L.fz, Cl.nz, L.pz != 0) << 18;
          e.w = addr(Cl, v[0] / L.fx, v[1] / L.fy, v[2] / L.fz);
          tab.push_back(e);
        }
  }
  for (int l = mg.tail; l < n - 1; ++l) {  // 1/diag and diag by row class
    const MgLevel &L = mg.lev[l];
    float2 d[kTailDiag] = {};
    for (int c = 0; c < 27; ++c) {
      const float dxy = L.wx * (float)(c / 9) + L.wy * (float)(c / 3 % 3);  // the products are exact
      d[c] = make_float2(L.idg[c], dxy + L.wz * (float)(c % 3));
    }
    const size_t at = tab.size();
    tab.resize(at + kTailDiag / 2);
    std::memcpy(&tab[at], d, sizeof d);
  }
  return tab;
}

template <typename T>
static void level_geometry(MgLevelT<T> &L, int nsm, bool quads) {
  L.bx = 1;
  while (L.bx < L.nz && L.bx < 32) L.bx *= 2;
  L.by = kBlock / L.bx;
  L.gx = (L.nz + L.bx - 1) / L.bx;
  L.gy = (L.ny + L.by - 1) / L.by;
  L.gz = std::max(1, std::min(L.nx, nsm * 8 / std::max(1, L.gx * L.gy)));
  // the quad smoother is FP32 (float4 loads): quads along x, rows along y, planes over z
  // (FP64: the pair passes, pairs along x)
  const bool pairs = sizeof(T) == sizeof(double) && L.nz % 2 == 0;
  L.qgrid = (quads && sizeof(T) == sizeof(float) && L.nz % 4 == 0) || pairs ? 1 : 0;
  if (L.qgrid) {
    const int nq = pairs ? L.nz / 2 : L.nz / 4;
    L.qbx = 1;
    while (L.qbx < nq && L.qbx < 32) L.qbx *= 2;
    L.qby = kBlock / L.qbx;
    L.qgx = (nq + L.qbx - 1) / L.qbx;
    L.qgy = (L.ny + L.qby - 1) / L.qby;
    L.qgz = std::max(1, std::min(L.nx, nsm * 8 / std::max(1, L.qgx * L.qgy)));
  }
}

// The marching kernels' bands and segments: the fewest units of time over the waves of blocks,
// each of msx planes, four halo planes and a start-up of about one, a plane costing a fixed part
// (the barrier and the latencies of one thread's chain) and one per thread of the
// multiprocessor: 0.74 us at 384 threads, 0.83 at 448 and 0.94 at 512 on 512x256x64.  Two blocks
// of up to 256 threads share one (128 registers a thread).  512x256x64: 29 x 5 blocks of 448 threads, one wave.
template <typename T>
static void march_geometry(MgLevelT<T> &L, int nsm) {
  const int nq = L.nz / 4, rows = L.ny / 2, most = kMgMarchThreads / nq - 2;
  const int b0 = (rows + most - 1) / most;
  double best = 0.0;
  for (int bands = b0; bands <= std::min(rows, b0 + 8); ++bands) {
    const int pairs = (rows + bands - 1) / bands, t = nq * (pairs + 2), per = t <= kMgMarchThreads / 2 ? 2 : 1;
    const int mgy = (rows + pairs - 1) / pairs;
    if (t < 64 && bands > b0) break;
    for (int segs = 1; segs <= L.nx / 2; ++segs) {
      const int msx = 2 * ((L.nx / 2 + segs - 1) / segs), mgx = (L.nx + msx - 1) / msx;
      const long long blocks = (long long)mgx * mgy, sm = (long long)per * nsm, waves = (blocks + sm - 1) / sm;
      const double on = (double)std::min<long long>(per, (blocks + nsm - 1) / nsm);  // blocks of a multiprocessor
      const double cost = (double)waves * (msx + 5) * (250.0 + on * t);
      if (best > 0.0 && cost >= best) continue;
      best = cost;
      L.mty = 2 * pairs;
      L.mgy = mgy;
      L.msx = msx;
      L.mgx = mgx;
    }
  }
  L.march = 1;
}

template <typename T>
bool mg_plan(int nx, int ny, int nz, double hx, double hy, double hz, int nsm, bool quads, MgPlanT<T> *mg,
             bool pz) {
  *mg = MgPlanT<T>{};
  int l = 0;
  for (;;) {
    MgLevelT<T> &L = mg->lev[l];
    L.nx = nx;
    L.ny = ny;
    L.nz = nz;
    L.pz = pz ? 1 : 0;
    // periodic z: red-black colouring holds across the wrap only for an even nz (or one
    // cell, which has no z neighbours)
    if (pz && nz % 2 && nz > 1) return false;
    L.wx = (T)(1.0 / (hx * hx));
    L.wy = (T)(1.0 / (hy * hy));
    L.wz = (T)(1.0 / (hz * hz));
    for (int q = 0; q < 27; ++q) {  // the diagonal as ldiag sums it, then its reciprocal
      const T d = L.wx * (T)(q / 9) + L.wy * (T)((q / 3) % 3) + L.wz * (T)(q % 3);
      L.idg[q] = d > T(0) ? T(1) / d : T(0);
    }
    level_geometry(L, nsm, quads);
    div_magic((unsigned)nz, &L.dz_m, &L.dz_l);
    div_magic((unsigned)ny, &L.dy_m, &L.dy_l);
    div_magic((unsigned)std::max(1, nz / 2), &L.dh_m, &L.dh_l);
    const long long cells = (long long)nx * ny * nz;
    const int fx = nx % 2 == 0 ? 2 : 1, fy = ny % 2 == 0 ? 2 : 1, fz = nz % 2 == 0 ? 2 : 1;
    if (cells <= kMgCoarseCells || fx * fy * fz == 1 || l + 1 == kMgMaxLevels) {
      L.fx = L.fy = L.fz = 1;
      break;
    }
    L.fx = fx;
    L.fy = fy;
    L.fz = fz;
    if (sizeof(T) == sizeof(float) && L.qgrid && fx == 2 && fy == 2 && fz == 2 && nz / 4 <= kMgMarchQuads &&
        cells < (1LL << 31))
      march_geometry(L, nsm);
    nx /= fx;
    ny /= fy;
    nz /= fz;
    hx *= fx;
    hy *= fy;
    hz *= fz;
    ++l;
  }
  mg->nlev = l + 1;
  // first level of the one-block tail: the smallest t >= 1 whose levels t..nlev-1 fit
  mg->tail = mg->nlev;  // none
  long long tail_cells = 0;
  for (int t = mg->nlev - 1; t >= 1; --t) {
    tail_cells += (long long)mg->lev[t].nx * mg->lev[t].ny * mg->lev[t].nz;
    if (tail_cells > tail_cells_max<T>()) break;
    mg->tail = t;
  }
  const MgLevelT<T> &C = mg->lev[l];
  mg->coarse_sweeps = std::min(256, 16 + 2 * std::max(C.nx, std::max(C.ny, C.nz)));
  return (long long)C.nx * C.ny * C.nz <= kMgSharedCells;
}

// per level above the tail (or the coarsest): 2 smooths + restrict, prolong + 2 smooths, or
// the two marching kernels; then one tail (or coarsest) kernel.  The FP64 pair passes start
// Jacobi-scaled rows (level 0) with one pass.
template <typename T>
int mg_vcycle_launches(const MgPlanT<T> &mg, int jacobi) {
  const int m = mg.tail < mg.nlev ? mg.tail : mg.nlev - 1;
  int n = 1;
  for (int l = 0; l < m; ++l) n += mg.lev[l].march ? 2 : 6;
  if (sizeof(T) == sizeof(double) && m > 0 && mg.lev[0].qgrid && jacobi) --n;
  return n;
}

// The pseudo-inverse of the coarsest level's operator (symmetric, singular on constants
// only): A+ = (A + J/n)^-1 - J/n with J the all-ones matrix, inverted by Gauss-Jordan with
// partial pivoting in double.  False when the level is larger than kMgDenseCells.
template <typename T>
bool mg_dense_inverse(const MgPlanT<T> &mg, std::vector<T> &M) {
  const MgLevelT<T> &C = mg.lev[mg.nlev - 1];
  const int n = C.nx * C.ny * C.nz;
  if (n > kMgDenseCells) return false;
  std::vector<double> A((size_t)n * n, 0.0), I((size_t)n * n, 0.0);
  const double wx = (double)C.wx, wy = (double)C.wy, wz = (double)C.wz;
  for (int i = 0; i < C.nx; ++i)
    for (int j = 0; j < C.ny; ++j)
      for (int k = 0; k < C.nz; ++k) {
        const int r = (i * C.ny + j) * C.nz + k;
        auto link = [&](int q, double w) {
          A[(size_t)r * n + q] -= w;
          A[(size_t)r * n + r] += w;
        };
        if (i > 0) link(r - C.ny * C.nz, wx);
        if (i < C.nx - 1) link(r + C.ny * C.nz, wx);
        if (j > 0) link(r - C.nz, wy);
        if (j < C.ny - 1) link(r + C.nz, wy);
        if (C.pz) {
          if (C.nz > 1) {
            link(k > 0 ? r - 1 : r + C.nz - 1, wz);
            link(k < C.nz - 1 ? r + 1 : r + 1 - C.nz, wz);
          }
        } else {
          if (k > 0) link(r - 1, wz);
          if (k < C.nz - 1) link(r + 1, wz);
        }
      }
  for (size_t q = 0; q < A.size(); ++q) A[q] += 1.0 / n;
  for (int r = 0; r < n; ++r) I[(size_t)r * n + r] = 1.0;
  for (int col = 0; col < n; ++col) {
    int piv = col;
    for (int r = col + 1; r < n; ++r)
      if (std::fabs(A[(size_t)r * n + col]) > std::fabs(A[(size_t)piv * n + col])) piv = r;
    if (!(std::fabs(A[(size_t)piv * n + col]) > 0.0)) return false;
    if (piv != col)
      for (int c = 0; c < n; ++c) {
        std::swap(A[(size_t)piv * n + c], A[(size_t)col * n + c]);
        std::swap(I[(size_t)piv * n + c], I[(size_t)col * n + c]);
      }
    const double inv = 1.0 / A[(size_t)col * n + col];
    for (int c = 0; c < n; ++c) {
      A[(size_t)col * n + c] *= inv;
      I[(size_t)col * n + c] *= inv;
    }
    for (int r = 0; r < n; ++r) {
      if (r == col) continue;
      const double f = A[(size_t)r * n + col];
      if (f == 0.0) continue;
      for (int c = 0; c < n; ++c) {
        A[(size_t)r * n + c] -= f * A[(size_t)col * n + c];
        I[(size_t)r * n + c] -= f * I[(size_t)col * n + c];
      }
    }
  }
  M.resize((size_t)n * n);
  for (int r = 0; r < n; ++r)
    for (int c = 0; c < n; ++c) M[(size_t)c * n + r] = (T)(I[(size_t)r * n + c] - 1.0 / n);
  return true;
}

template <typename T>
void mg_prepare() {
  // the one-block kernels of the FP64 hierarchy need more than the default 48 KB
  cudaFuncSetAttribute(k_mg_coarse<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(2 * sizeof(T) * kMgSharedCells));
  cudaFuncSetAttribute(k_mg_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMgTailBytes);
  if (sizeof(T) == sizeof(float))
    cudaFuncSetAttribute(k_mg_tail32, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailShared);
}

template <typename T>
void launch_mg_vcycle(cudaStream_t s, const MgPlanT<T> &mg, int jacobi, const T *b0, T *x0, const SolverScal *sc) {
  const int n = mg.nlev;
  auto B = [&](int l) -> const T * { return l == 0 ? b0 : mg.lev[l].b; };
  auto X = [&](int l) -> T * { return l == 0 ? x0 : mg.lev[l].x; };
  auto grid = [&](int l) { return dim3(mg.lev[l].gx, mg.lev[l].gy, mg.lev[l].gz); };
  auto block = [&](int l) { return dim3(mg.lev[l].bx, mg.lev[l].by, 1); };
  auto smooth = [&](int l, int colour, int zero) {
    if constexpr (sizeof(T) == sizeof(float)) {
      if (mg.lev[l].qgrid > 0) {
        const MgLevelT<T> &Q = mg.lev[l];
        launch_pdl(k_mg_smooth4, dim3(Q.qgx, Q.qgy, Q.qgz), dim3(Q.qbx, Q.qby, 1), 0, s, Q, colour, zero,
                   l == 0 ? jacobi : 0, B(l), X(l), sc);
        return;
      }
    }
    launch_pdl(k_mg_smooth<T>, grid(l), block(l), 0, s, mg.lev[l], colour, zero, l == 0 ? jacobi : 0, B(l), X(l), sc);
  };
  // a colour pass of the FP64 pair kernels
  auto pair = [&](int l, int colour, int from_b) {
    if constexpr (sizeof(T) == sizeof(double)) {
      const MgLevelT<T> &F = mg.lev[l];
      launch_pdl(l == 0 && jacobi ? k_mgp_colour<true> : k_mgp_colour<false>, dim3(F.qgx, F.qgy, F.qgz),
                 dim3(F.qbx, F.qby, 1), 0, s, F, colour, from_b, B(l), X(l), sc);
    }
  };
  // pre-smoothing from zero and restriction to level l + 1.  (Both colour passes in one
  // kernel, each black cell recomputing its red neighbours' start values, was measured at
  // 80 us on the 512x256x64 level against 36 us for the two quad passes: not kept.)
  // the marching kernels of a level (FP32 only)
  auto march = [&](int l, bool up) {
    if constexpr (sizeof(T) == sizeof(float)) {
      const MgLevelT<T> &F = mg.lev[l], &Cl = mg.lev[l + 1];
      const bool bs = l == 0 && jacobi;
      const dim3 grid(F.mgx, F.mgy), block(F.nz / 4 * (F.mty / 2 + 2));
      if (up)
        launch_pdl(bs ? k_mg_up<true> : k_mg_up<false>, grid, block, 0, s, F, Cl, B(l), (const T *)X(l + 1), X(l), sc);
      else
        launch_pdl(bs ? k_mg_down<true> : k_mg_down<false>, grid, block, 0, s, F, Cl, B(l), Cl.b, sc);
    }
  };
  auto down = [&](int l) {
    if (mg.lev[l].march) {
      march(l, false);
      return;
    }
    const int bs = l == 0 ? jacobi : 0;
    const MgLevelT<T> &F = mg.lev[l];
    if constexpr (sizeof(T) == sizeof(double)) {
      if (F.qgrid) {
        if (!bs)
          launch_pdl(k_mgp_scale, dim3(F.qgx, F.qgy, F.qgz), dim3(F.qbx, F.qby, 1), 0, s, F, B(l), X(l), sc);
        pair(l, 1, bs);
        if (F.fx == 2 && F.fy == 2 && F.fz == 2)
          launch_pdl(k_mgp_restrict, grid(l + 1), block(l + 1), 0, s, F, mg.lev[l + 1], (const T *)X(l),
                     mg.lev[l + 1].b, sc);
        else
          launch_pdl(k_mg_restrict<T>, grid(l + 1), block(l + 1), 0, s, F, mg.lev[l + 1], bs, B(l), X(l),
                     mg.lev[l + 1].b, sc);
        return;
      }
    }
    smooth(l, 0, 1);
    smooth(l, 1, 0);
    if (F.fx == 2 && F.fy == 2 && F.fz == 2)
      launch_pdl(k_mg_restrict8<T>, grid(l + 1), block(l + 1), 0, s, F, mg.lev[l + 1], bs, B(l), X(l),
                 mg.lev[l + 1].b, sc);
    else
      launch_pdl(k_mg_restrict<T>, grid(l + 1), block(l + 1), 0, s, F, mg.lev[l + 1], bs, B(l), X(l),
                 mg.lev[l + 1].b, sc);
  };
  const int m = std::min(mg.tail, n);  // levels m..n-1 run in one block (m < n), or none
  for (int l = 0; l + 1 < m; ++l) down(l);
  if (m < n) {
    down(m - 1);  // levels m-1 -> m as above, then the tail
    size_t cells = 0, bytes = 0;
    for (int l = m; l < n; ++l) cells += (size_t)mg.lev[l].nx * mg.lev[l].ny * mg.lev[l].nz;
    if constexpr (sizeof(T) == sizeof(float)) {
      if (mg.ttab) {
        const TailLayout o = tail_layout(mg);
        bytes = 4 * (size_t)o.words;
        launch_pdl(k_mg_tail32, dim3(1), dim3(1024), bytes, s, mg, o, sc);
      }
    }
    if (bytes == 0) launch_pdl(k_mg_tail<T>, dim3(1), dim3(1024), 2 * sizeof(T) * cells, s, mg, m, sc);
  } else {
    const MgLevelT<T> &C = mg.lev[n - 1];
    const size_t smem = 2 * sizeof(T) * (size_t)C.nx * C.ny * C.nz;
    launch_pdl(k_mg_coarse<T>, dim3(1), dim3(1024), smem, s, C, mg.coarse_sweeps, mg.cinv, n == 1 ? jacobi : 0,
               B(n - 1), X(n - 1), sc);
  }
  for (int l = (m < n ? m : n - 1) - 1; l >= 0; --l) {
    const MgLevelT<T> &F = mg.lev[l];
    if (F.march) {
      march(l, true);
      continue;
    }
    if constexpr (sizeof(T) == sizeof(double)) {
      if (F.qgrid) {
        if (F.fx == 2 && F.fy == 2 && F.fz == 2)
          launch_pdl(k_mgp_prolong, grid(l + 1), block(l + 1), 0, s, F, mg.lev[l + 1], (const T *)X(l + 1), X(l), sc);
        else
          launch_pdl(k_mg_prolong<T>, grid(l), block(l), 0, s, F, mg.lev[l + 1], (const T *)X(l + 1), X(l), sc);
        pair(l, 1, 0);
        pair(l, 0, 0);
        continue;
      }
    }
    if (F.fx == 2 && F.fy == 2 && F.fz == 2)
      launch_pdl(k_mg_prolong8<T>, grid(l + 1), block(l + 1), 0, s, F, mg.lev[l + 1], (const T *)X(l + 1), X(l), sc);
    else
      launch_pdl(k_mg_prolong<T>, grid(l), block(l), 0, s, F, mg.lev[l + 1], (const T *)X(l + 1), X(l), sc);
    smooth(l, 1, 0);
    smooth(l, 0, 0);
  }
}

template bool mg_plan<float>(int, int, int, double, double, double, int, bool, MgPlanT<float> *, bool);
template bool mg_plan<double>(int, int, int, double, double, double, int, bool, MgPlanT<double> *, bool);
template int mg_vcycle_launches<float>(const MgPlanT<float> &, int);
template bool mg_dense_inverse<float>(const MgPlanT<float> &, std::vector<float> &);
template bool mg_dense_inverse<double>(const MgPlanT<double> &, std::vector<double> &);
template int mg_vcycle_launches<double>(const MgPlanT<double> &, int);
template void mg_prepare<float>();
template void mg_prepare<double>();
template void launch_mg_vcycle<float>(cudaStream_t, const MgPlanT<float> &, int, const float *, float *,
                                      const SolverScal *);
template void launch_mg_vcycle<double>(cudaStream_t, const MgPlanT<double> &, int, const double *, double *,
                                       const SolverScal *);

}  // namespace cfdgb
