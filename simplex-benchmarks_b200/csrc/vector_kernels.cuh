// Vector kernels of the solvers and the multigrid cycle (FP64 and FP32).
//
// These replace the deal.II LinearAlgebra::distributed::Vector operations
// used by SolverCG, PreconditionChebyshev and MGTransferGlobalCoarsening
// (add/sadd/equ/scale, dot products, norms).  Reductions are two-stage with a
// fixed block order, so results are bitwise reproducible.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "pdl.cuh"

namespace sfem {

constexpr int kReduceBlocks = 592;  // 4 x 148 SMs
constexpr int kReduceThreads = 256;

template <typename To, typename Ti>
__global__ void vec_convert(int64_t n, const Ti* __restrict__ in, To* __restrict__ out) {
  pdl_enter();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = To(in[i]);
}

// y = a x + b y
template <typename T>
__global__ void vec_axpby(int64_t n, T a, const T* __restrict__ x, T b, T* __restrict__ y) {
  pdl_enter();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    y[i] = a * x[i] + b * y[i];
}

// v with its bits and-ed with mask (0 in every call: the result is 0).  A kernel
// that clears a value it has read stores this instead of a constant, so that the
// store waits for the load: a store that is issued while a load of its line is
// outstanding is very slow (Chebyshev step on 7.2M FP32 values, B200: 290 us
// with a constant, 45 us with the masked value, 41 us without the store).
__device__ __forceinline__ float cleared(float v, int mask) { return __int_as_float(__float_as_int(v) & mask); }
__device__ __forceinline__ double cleared(double v, int mask) {
  return __longlong_as_double(__double_as_longlong(v) & (long long)(mask));
}

// r = b - t.  ZERO: t = 0 after it has been read (the next product adds into
// it), and z[0 .. nz) = 0 (the coarse right-hand side the residual is restricted
// into): two fills without launches of their own.
template <typename T, bool ZERO = false>
__global__ void vec_residual(int64_t n, const T* __restrict__ b, T* __restrict__ t, T* __restrict__ r,
                             T* __restrict__ z, int64_t nz, int mask) {
  pdl_enter();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const T ti = t[i];
    r[i] = b[i] - ti;
    if (ZERO) t[i] = cleared(ti, mask);
  }
  if (z)
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < nz; i += int64_t(gridDim.x) * blockDim.x)
      z[i] = T(0);
}

// z = invd .* r
template <typename T>
__global__ void vec_scale(int64_t n, const T* __restrict__ invd, const T* __restrict__ r, T* __restrict__ z) {
  pdl_enter();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    z[i] = invd[i] * r[i];
}

// Two-stage sum over the grid in one launch: every block leaves its sum (fixed
// order inside the block), the last one to arrive adds the blocks' sums in order
// and clears the counter for the next launch.  Results do not depend on which
// block that is.  scratch: kReduceBlocks sums, then the arrival counter (zero).
__device__ __forceinline__ void grid_sum(double acc, double* scratch, double* out) {
  __shared__ double s[kReduceThreads];
  __shared__ bool last;
  unsigned* count = reinterpret_cast<unsigned*>(scratch + kReduceBlocks);
  auto block_sum = [&](double v) {
    s[threadIdx.x] = v;
    __syncthreads();
    for (int w = kReduceThreads / 2; w > 0; w >>= 1) {
      if (int(threadIdx.x) < w) s[threadIdx.x] += s[threadIdx.x + w];
      __syncthreads();
    }
    return s[0];
  };
  const double b = block_sum(acc);
  if (threadIdx.x == 0) {
    scratch[blockIdx.x] = b;
    __threadfence();
    last = atomicAdd(count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v = 0.0;
  for (int i = threadIdx.x; i < int(gridDim.x); i += kReduceThreads) v += __ldcg(scratch + i);
  __syncthreads();
  const double total = block_sum(v);
  if (threadIdx.x == 0) {
    *out = total;
    *count = 0;
  }
}
constexpr size_t kReduceScratch = kReduceBlocks + 1;  // doubles, zero at first

// *out = x . y (double accumulation); launched with kReduceBlocks x kReduceThreads
template <typename T>
__global__ void __launch_bounds__(kReduceThreads) vec_dot(int64_t n, const T* __restrict__ x,
                                                          const T* __restrict__ y, double* __restrict__ scratch,
                                                          double* __restrict__ out) {
  pdl_enter();
  double acc = 0.0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    acc += double(x[i]) * double(y[i]);
  grid_sum(acc, scratch, out);
}

// W values moved at once: 16 bytes on large aligned vectors, else one.  The
// Chebyshev steps of large levels are bound by memory and by how much of it a thread
// asks for: 64^3 P3 solve, B200, 13.3 -> 13.07 ms.  The same in the dot products and CG
// updates gained 0.4 % and is not done.
template <typename T, int W>
struct alignas(W * sizeof(T)) Pack {
  T v[W];
};
template <typename T, int W>
__device__ __forceinline__ Pack<T, W> pack_at(const T* p, int64_t i) {
  return reinterpret_cast<const Pack<T, W>*>(p)[i];
}

// Chebyshev, first step from a zero initial guess: d = c P b, x = d
template <typename T, int W>
__global__ void cheb_first_zero(int64_t n, T c, const T* __restrict__ invd, const T* __restrict__ b,
                                T* __restrict__ d, T* __restrict__ x) {
  pdl_enter();
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x, nw = n / W;
  for (int64_t i = t; i < nw; i += int64_t(gridDim.x) * blockDim.x) {
    const Pack<T, W> bi = pack_at<T, W>(b, i), pi = pack_at<T, W>(invd, i);
    Pack<T, W> v;
#pragma unroll
    for (int k = 0; k < W; ++k) v.v[k] = c * pi.v[k] * bi.v[k];
    reinterpret_cast<Pack<T, W>*>(d)[i] = v;
    reinterpret_cast<Pack<T, W>*>(x)[i] = v;
  }
  if (W > 1 && t < n - nw * W) {
    const int64_t i = nw * W + t;
    const T v = c * invd[i] * b[i];
    d[i] = v;
    x[i] = v;
  }
}

// Chebyshev step: d = f1 d + f2 P (b - t), x += d   (t = A x); FIRST: the
// first step from a nonzero x, d = f2 P (b - t) (d is not read); ZERO (W = 1): t = 0
// after it has been read (the next product adds into it)
template <typename T, bool FIRST, bool ZERO, int W>
__global__ void cheb_step(int64_t n, T f1, T f2, const T* __restrict__ invd, const T* __restrict__ b,
                          T* __restrict__ t, T* __restrict__ d, T* __restrict__ x, int mask) {
  static_assert(!ZERO || W == 1, "the clearing form goes value by value");
  pdl_enter();
  const int64_t t0 = blockIdx.x * int64_t(blockDim.x) + threadIdx.x, nw = n / W;
  for (int64_t i = t0; i < nw; i += int64_t(gridDim.x) * blockDim.x) {
    const Pack<T, W> ti = pack_at<T, W>(t, i), bi = pack_at<T, W>(b, i), pi = pack_at<T, W>(invd, i);
    Pack<T, W> di, xi = pack_at<T, W>(x, i);
    if (!FIRST) di = pack_at<T, W>(d, i);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      di.v[k] = (FIRST ? T(0) : f1 * di.v[k]) + f2 * pi.v[k] * (bi.v[k] - ti.v[k]);
      xi.v[k] += di.v[k];
    }
    reinterpret_cast<Pack<T, W>*>(d)[i] = di;
    reinterpret_cast<Pack<T, W>*>(x)[i] = xi;
    if (ZERO) t[i] = cleared(ti.v[0], mask);
  }
  if (W > 1 && t0 < n - nw * W) {
    const int64_t i = nw * W + t0;
    const T v = (FIRST ? T(0) : f1 * d[i]) + f2 * invd[i] * (b[i] - t[i]);
    d[i] = v;
    x[i] += v;
  }
}

// y = A x for a small dense FP64 matrix (coarse-grid solve), one warp per row
template <typename T>
__global__ void dense_matvec(int n, const double* __restrict__ A, const T* __restrict__ x, T* __restrict__ y) {
  pdl_enter();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n) return;
  double acc = 0.0;
  for (int j = lane; j < n; j += 32) acc += A[int64_t(warp) * n + j] * double(x[j]);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) y[warp] = T(acc);
}

// CG update with the step read on the device: alpha = sc[rz] / sc[pq];
// nothing is updated unless sc[pq] is finite and positive (the host reads
// sc[pq] after the step and reports the breakdown).  sc[rr] = (r, r) of the new
// residual (of the old one after a breakdown).  ZERO: q = 0 after it has been
// read (the next product adds into it).  Launched with kReduceBlocks x kReduceThreads.
template <bool ZERO>
__global__ void __launch_bounds__(kReduceThreads) cg_update_xr(int64_t n, double* sc, int rz, int pq, int rr,
                                                               const double* __restrict__ p, double* __restrict__ q,
                                                               double* __restrict__ x, double* __restrict__ r,
                                                               double* __restrict__ scratch, int mask) {
  pdl_enter();
  const double den = sc[pq];
  const bool ok = den > 0 && isfinite(den);
  const double alpha = ok ? sc[rz] / den : 0.0;
  double acc = 0.0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    double ri = r[i];
    const double qi = q[i];
    if (ok) {
      x[i] += alpha * p[i];
      ri -= alpha * qi;
      r[i] = ri;
    }
    if (ZERO) q[i] = cleared(qi, mask);
    acc += ri * ri;
  }
  grid_sum(acc, scratch, sc + rr);
}

// p = a z + beta p with beta = (sc[num] - (sub >= 0 ? sc[sub] : 0)) / sc[den], read on the device
static __global__ void cg_update_p_dev(int64_t n, double a, const double* __restrict__ sc, int num, int sub, int den,
                                       const double* __restrict__ z, double* __restrict__ p) {
  pdl_enter();
  const double beta = (sub >= 0 ? sc[num] - sc[sub] : sc[num]) / sc[den];
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    p[i] = a * z[i] + beta * p[i];
}

// x += (sc[0]/sc[1]) z  (step 0 unless sc[1] > 0); the ratio stays on the device
template <typename T>
__global__ void axpy_ratio(int64_t n, const double* __restrict__ sc, const T* __restrict__ z, T* __restrict__ x) {
  pdl_enter();
  const double den = sc[1];
  const T w = den > 0.0 ? T(sc[0] / den) : T(0);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    x[i] += w * z[i];
}

// r = b - (sc[0]/sc[1]) q
template <typename T>
__global__ void residual_ratio(int64_t n, const double* __restrict__ sc, const T* __restrict__ b,
                               const T* __restrict__ q, T* __restrict__ r) {
  pdl_enter();
  const double den = sc[1];
  const T w = den > 0.0 ? T(sc[0] / den) : T(0);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    r[i] = b[i] - w * q[i];
}

// 16 bytes at once: vectors that fill the SMs so, at 16-byte addresses
template <typename T>
inline bool in_packs(int64_t n, const T* x, const T* y) {
  return n >= 148 * 2048 * int64_t(16 / sizeof(T)) &&
         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0;
}
inline unsigned grid_for(int64_t n, int bs = 256, unsigned cap = 148 * 16) {
  const int64_t b = (n + bs - 1) / bs;
  return unsigned(b < cap ? (b > 0 ? b : 1) : cap);
}

}  // namespace sfem
