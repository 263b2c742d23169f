// Deterministic two-stage FP64 reductions for kernels with a fixed grid (1-D or 3-D
// blocks of kBlock threads).
//
// Stage 1: each block reduces its NV per-thread values (warp shuffles + shared memory)
// and stores them to part[q * nblocks + block].  Stage 2: the last block to finish (atomic
// ticket) sums the partials in a fixed order, so results do not depend on block
// scheduling.  No block ever waits on another.
#pragma once

#include "cfdgb_internal.cuh"

namespace cfdgb {

__device__ __forceinline__ int lin_tid() { return (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int lin_bid() { return (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x; }
__device__ __forceinline__ int nblocks() { return gridDim.x * gridDim.y * gridDim.z; }

// Sum of a value over the warp, in every lane.  The FP64 pipe issues one warp instruction
// per 64 cycles and scheduler whatever the lanes do (measured: 2.0 lanes per cycle and SM,
// predicated off or not), so a shuffle tree costs 5 x 64 cycles of it per warp and value:
// on a grid of a few cells a thread, more than the dot product that it ends.  Here the values
// are added as integers instead: each mantissa, shifted to the warp's largest exponent (4
// bits below its last place kept, rounded), is split into 26-bit fields whose sums over 32
// lanes fit 32 bits (three redux.sync), and the total is converted back once.  The rounding
// is at most 1/32 ulp of the largest value per lane, below that of a tree of FP64 additions,
// and the result does not depend on the order.  With the scalar work on three lanes (div3), on the
// kernels a phase: FP64 BiCGSTAB on 256x128x32 88 -> 74 us an iteration, FP64 CG on 151x77x27 29.5 -> 24.3,
// FP32 CG sweeps on 256x128x64 24.0 -> 21.5.  Values that do not fit this (Inf, NaN, and
// exponents near either end of the range) take the shuffle tree.
constexpr int kSumGuard = 4;  // bits kept below the largest value's last place
__device__ __forceinline__ double warp_sum1(double v) {
  const long long b = __double_as_longlong(v);
  const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
  const unsigned em = __reduce_max_sync(0xffffffffu, e);
  if (em - 96u <= 0x7f0u - 96u) {  // 96 <= em <= 0x7f0, the same in every lane
    const unsigned s = em - e;     // zeros and subnormals: s >= 95, nothing left after the shift
    const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffULL) | 0x10000000000000ULL;
    const unsigned long long r = s < 64u ? ((m << kSumGuard) + ((1ULL << s) >> 1)) >> s : 0ULL;
    const long long f = b < 0 ? -(long long)r : (long long)r;
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)f & 0x3ffffffu);
    const unsigned mi = __reduce_add_sync(0xffffffffu, (unsigned)(f >> 26) & 0x3ffffffu);
    const int hi = __reduce_add_sync(0xffffffffu, (int)(f >> 52));
    const long long t = ((long long)hi << 52) + ((long long)mi << 26) + (long long)lo;  // |t| < 2^62
    if (t == 0) return 0.0;
    return __longlong_as_double(__double_as_longlong((double)t) + ((long long)((int)em - 1075 - kSumGuard) << 52));
  }
  if (!__any_sync(0xffffffffu, !is_zero(v))) return 0.0;  // drag sums away from the body
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

template <int NV>
__device__ __forceinline__ void warp_sum(double (&v)[NV]) {
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = warp_sum1(v[q]);
}

// Reduce v over the block (whole warps, at most 32 of them); the result is valid in
// thread 0 only.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
  __shared__ double sh[NV][32];
  const int t = lin_tid();
  const int lane = t & 31, wid = t >> 5;
  const int nw = (int)(blockDim.x * blockDim.y * blockDim.z) >> 5;
  warp_sum<NV>(v);
  __syncthreads();  // sh may still be read by a previous call
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) sh[q][wid] = v[q];
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = lane < nw ? sh[q][lane] : 0.0;
    warp_sum<NV>(v);
  }
}

// Stage 1 + 2.  Returns true in every thread of the last block; out[] is then valid in
// all of its threads.  *ticket is reset for the next launch.
template <int NV>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], double *part, unsigned *ticket,
                                         double (&out)[NV]) {
  __shared__ bool last;
  __shared__ double res[NV];
  block_sum<NV>(v);
  const int G = nblocks(), t = lin_tid();
  if (t == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) part[q * G + lin_bid()] = v[q];
    __threadfence();
    last = (atomicAdd(ticket, 1u) == (unsigned)(G - 1));
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double w[NV];
  const int nt = (int)(blockDim.x * blockDim.y * blockDim.z);
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double s = 0.0;
    for (int b = t; b < G; b += nt) s += __ldcg(part + q * G + b);
    w[q] = s;
  }
  block_sum<NV>(w);
  if (t == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) res[q] = w[q];
    *ticket = 0u;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) out[q] = res[q];
  return true;
}

// The larger of two doubles on the integer pipe (an FP64 comparison takes the FP64 pipe, see
// warp_sum1): ordered 64-bit keys, a NaN never taken over a number (as fmax).
__device__ __forceinline__ double max_int(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  const long long kx = x ^ ((x >> 63) & 0x7fffffffffffffffLL), ky = y ^ ((y >> 63) & 0x7fffffffffffffffLL);
  const bool nan = (__double2hiint(b) & 0x7fffffff) >= 0x7ff80000;
  return ky > kx && !nan ? b : a;
}

// Grid-wide maxima of NV values per thread (no NaN among them), with the same last-block
// pattern as grid_sum (minima: pass the negated values).  Maxima are exact, so the result
// does not depend on the order either.
template <int NV>
__device__ __forceinline__ void block_max(double (&v)[NV], double (*sh)[32]) {
  const int t = lin_tid(), lane = t & 31, wid = t >> 5;
  const int nw = (int)(blockDim.x * blockDim.y * blockDim.z) >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[q] = max_int(v[q], __shfl_xor_sync(0xffffffffu, v[q], off));
  __syncthreads();  // sh may still be read by a previous call
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) sh[q][wid] = v[q];
  __syncthreads();
  if (wid == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      v[q] = lane < nw ? sh[q][lane] : -INFINITY;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v[q] = max_int(v[q], __shfl_xor_sync(0xffffffffu, v[q], off));
    }
}
template <int NV>
__device__ __forceinline__ bool grid_max(double (&v)[NV], double *part, unsigned *ticket, double (&out)[NV]) {
  __shared__ double sh[NV][32];
  __shared__ bool last;
  __shared__ double res[NV];
  block_max<NV>(v, sh);
  const int G = nblocks(), t = lin_tid();
  if (t == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) part[q * G + lin_bid()] = v[q];
    __threadfence();
    last = (atomicAdd(ticket, 1u) == (unsigned)(G - 1));
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int nt = (int)(blockDim.x * blockDim.y * blockDim.z);
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double m = -INFINITY;
    for (int b = t; b < G; b += nt) m = max_int(m, __ldcg(part + q * G + b));
    v[q] = m;
  }
  block_max<NV>(v, sh);
  if (t == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) res[q] = v[q];
    *ticket = 0u;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) out[q] = res[q];
  return true;
}

// FP32 products summed in short FP32 runs, each run added into an FP64 accumulator:
// global sums stay FP64 while the per-element work stays FP32.
struct AccF {
  double d = 0.0;
  float f = 0.0f;
  int n = 0;
  __device__ __forceinline__ void add(float x) {
    f += x;
    if (++n == 8) { d += (double)f; f = 0.0f; n = 0; }
  }
  __device__ __forceinline__ double get() const { return d + (double)f; }
};
// Compensated FP32 dot product (Ogita, Rump and Oishi's Dot2: the error-free product by
// FMA and Knuth's TwoSum): as accurate as a dot product in twice the working precision,
// at a few FP32 operations per term.
struct Dot2F {
  float hi = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void add(float a, float b) {
    const float p = a * b;
    const float pe = fmaf(a, b, -p);  // a*b - p exactly
    const float s = hi + p;
    const float bp = s - hi;
    const float se = (hi - (s - bp)) + (p - bp);  // hi + p - s exactly
    hi = s;
    lo += pe + se;
  }
  __device__ __forceinline__ double get() const { return (double)hi + (double)lo; }
};
// Plain FP32 running sum of products for the vectorised kernels: a thread covers a few
// dozen quads, and the sum over threads is FP64 (grid_sum).
struct SumF {
  float f = 0.0f;
  __device__ __forceinline__ void add(float a, float b) { f = fmaf(a, b, f); }
  __device__ __forceinline__ double get() const { return (double)f; }
};
struct AccD {
  double d = 0.0;
  __device__ __forceinline__ void add(double x) { d += x; }
  __device__ __forceinline__ double get() const { return d; }
};
template <typename T> struct AccFor;
template <> struct AccFor<double> { using type = AccD; };
template <> struct AccFor<float> { using type = AccF; };

}  // namespace cfdgb
