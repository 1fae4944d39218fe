// Training gradient of the learned smoother's MLP: loss = mean_b ||o_b - y_b||^2
// and its derivative in every (BF16-rounded) parameter, FP32 throughout.
//
// One CTA of 256 threads takes tiles of S = 16 SPT samples and runs the three
// layers forward and backward on the whole tile from shared memory, as small
// matrix products: [S x 32] [32 x 64], [S x 64] [64 x 64], [S x 64] [64 x 20]
// and their transposes.  Activations are kept sample-major, the weights in both
// orientations, so that every product reads 16-byte rows: a thread owns four
// neighbouring outputs of SPT samples (or a 4 x 4 block of a weight gradient)
// and a warp's reads are broadcasts or contiguous rows without bank conflicts
// (row strides of 68 and 36 words).  The weight gradients stay in registers
// over all tiles of the CTA and leave once, as coalesced atomic additions in FP64
// that a second small launch rounds.  Added in FP32, one CTA's sums after another onto
// the same total (128 CTAs for 2048 samples), the gradient's error against 64 bits is
// 1.6e-7 at 2048 and 2.2e-7 at 8192 samples; so it is 3e-8 at both, for 2 us of a
// call.  Eight or four CTAs of a cluster adding pairwise before an FP32 addition leave
// 6e-8 and 8e-8, but 16 clusters of eight or more than 33 of four do not fit with one
// CTA per SM (51 us a call).  A workspace of one row per CTA would be reproducible bit
// for bit, but its allocation costs 3 ms on the first call.
//
// The kernel is bound by shared-memory reads (about 9 wavefronts for 16
// multiply-adds of a warp) and by the latency of the eight products of a tile;
// small batches are given one 16-sample tile per CTA to fill the SMs.  Measured
// on B200, the whole call with its host read of the loss: 2048 samples (the
// default batch) 33.8 us, 32,768 samples 95 us, against 13.1 and 13.7 ms for a
// thread per sample with shared-memory atomics for every product.  The rounding launch
// writes the loss to pinned memory; a copy after it would make that 40.7 us.
#pragma once
#include <cuda_bf16.h>

#include "mlp.cuh"
#include "mlp_dims.hpp"
#include "pdl.cuh"

namespace sfem {
namespace mlpg {

constexpr int THREADS = 256;
constexpr int HS = 68;  // row stride of hidden activations [S][64]
constexpr int XS = 36;  // row stride of inputs [S][32] (29 padded with zeros)

// shared memory, in floats
constexpr int O_W1T = 0;                        // [32][64] (rows 29..31 zero)
constexpr int O_W2T = O_W1T + 32 * 64;          // [64][64]
constexpr int O_W2 = O_W2T + 64 * 64;           // [64][64]
constexpr int O_W3T = O_W2 + 64 * 64;           // [64][20]
constexpr int O_W3 = O_W3T + 64 * 20;           // [20][64]
constexpr int O_B = O_W3 + 20 * 64;             // b1 [64], b2 [64], b3 [20]
constexpr int O_ACT = O_B + 148;
template <int SPT>
struct Shape {
  static constexpr int S = 16 * SPT;
  static constexpr int O_X = O_ACT;             // [S][XS]
  static constexpr int O_H1 = O_X + S * XS;     // [S][HS] activations of layer 1
  static constexpr int O_D1 = O_H1 + S * HS;    // their GELU derivative, then dLoss/da1
  static constexpr int O_H2 = O_D1 + S * HS;
  static constexpr int O_D2 = O_H2 + S * HS;
  static constexpr int O_DO = O_D2 + S * HS;    // [S][20] dLoss/do
  static constexpr int FLOATS = O_DO + S * 20;
  static constexpr size_t BYTES = sizeof(float) * FLOATS;
};

// GELU and its derivative with one tanh (the forms of gelu and gelu_grad)
__device__ __forceinline__ void gelu_both(float x, float& h, float& d) {
  const float t = tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x));
  h = 0.5f * x * (1.0f + t);
  d = 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * 0.7978845608028654f * (1.0f + 0.134145f * x * x);
}

__device__ __forceinline__ void fma4(float (&a)[4], const float4& w, float x) {
  a[0] = fmaf(w.x, x, a[0]);
  a[1] = fmaf(w.y, x, a[1]);
  a[2] = fmaf(w.z, x, a[2]);
  a[3] = fmaf(w.w, x, a[3]);
}

// acc[q][0..3] += sum_k M[k][4 col ..] v[s0 + 16 q][k], M with MC columns
template <int K, int MC, int VS, int SPT>
__device__ __forceinline__ void product(const float* M, const float* v, int col, int s0, float (&acc)[SPT][4]) {
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 x[SPT];
#pragma unroll
    for (int q = 0; q < SPT; ++q) x[q] = *reinterpret_cast<const float4*>(v + (s0 + 16 * q) * VS + k);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 w = *reinterpret_cast<const float4*>(M + (k + e) * MC + 4 * col);
#pragma unroll
      for (int q = 0; q < SPT; ++q) fma4(acc[q], w, e == 0 ? x[q].x : e == 1 ? x[q].y : e == 2 ? x[q].z : x[q].w);
    }
  }
}

}  // namespace mlpg

// sums [NPARAM] and loss are zero on entry (loss: or a running sum)
template <int SPT>
__global__ void __launch_bounds__(mlpg::THREADS, 2)
    mlp_grad_kernel(int n, const float* __restrict__ X, const float* __restrict__ Y,
                    const __nv_bfloat16* __restrict__ wb, double* __restrict__ sums, double* __restrict__ loss,
                    float inv_batch) {
  using D = MLPDims;
  using namespace mlpg;
  using Sh = Shape<SPT>;
  constexpr int S = Sh::S;
  extern __shared__ __align__(16) float sm[];
  const int t = threadIdx.x;
  // unrolled so that all of a thread's weight loads are in flight together
#pragma unroll
  for (int i = t; i < 32 * 64; i += THREADS)
    sm[O_W1T + i] = i / 64 < D::NIN ? __bfloat162float(wb[D::OFF_W1 + (i % 64) * D::NIN + i / 64]) : 0.0f;
#pragma unroll
  for (int i = t; i < 64 * 64; i += THREADS) {
    const float w = __bfloat162float(wb[D::OFF_W2 + i]);
    sm[O_W2 + i] = w;
    sm[O_W2T + (i % 64) * 64 + i / 64] = w;
  }
#pragma unroll
  for (int i = t; i < 20 * 64; i += THREADS) {
    const float w = __bfloat162float(wb[D::OFF_W3 + i]);
    sm[O_W3 + i] = w;
    sm[O_W3T + (i % 64) * 20 + i / 64] = w;
  }
  for (int i = t; i < 148; i += THREADS)
    sm[O_B + i] = __bfloat162float(wb[i < 64 ? D::OFF_B1 + i : i < 128 ? D::OFF_B2 + i - 64 : D::OFF_B3 + i - 128]);

  const int col = t & 15, s0 = t >> 4;   // products: outputs 4 col .. 4 col + 3 of samples s0 + 16 q
  const int gr = t >> 4, gc = t & 15;    // weight gradients: rows 4 gr .., columns 4 gc .. (2 gc .. for W1)
  float g1[4][2] = {}, g2[4][4] = {}, g3[5] = {}, gb = 0.0f, lsum = 0.0f;
  const int tiles = (n + S - 1) / S;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int b0 = tile * S;
    __syncthreads();  // the weights are staged; the previous tile is done with every buffer
#pragma unroll
    for (int i = t; i < S * 32; i += THREADS) {
      const int s = i / 32, k = i % 32;
      sm[Sh::O_X + s * XS + k] = (b0 + s < n && k < D::NIN) ? __ldg(X + int64_t(b0 + s) * D::NIN + k) : 0.0f;
    }
    __syncthreads();
    // ---- forward
    {
      float a[SPT][4];
#pragma unroll
      for (int q = 0; q < SPT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[q][e] = sm[O_B + 4 * col + e];
      product<32, 64, XS, SPT>(sm + O_W1T, sm + Sh::O_X, col, s0, a);
#pragma unroll
      for (int q = 0; q < SPT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          gelu_both(a[q][e], sm[Sh::O_H1 + (s0 + 16 * q) * HS + 4 * col + e],
                    sm[Sh::O_D1 + (s0 + 16 * q) * HS + 4 * col + e]);
    }
    __syncthreads();
    {
      float a[SPT][4];
#pragma unroll
      for (int q = 0; q < SPT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[q][e] = sm[O_B + 64 + 4 * col + e];
      product<64, 64, HS, SPT>(sm + O_W2T, sm + Sh::O_H1, col, s0, a);
#pragma unroll
      for (int q = 0; q < SPT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          gelu_both(a[q][e], sm[Sh::O_H2 + (s0 + 16 * q) * HS + 4 * col + e],
                    sm[Sh::O_D2 + (s0 + 16 * q) * HS + 4 * col + e]);
    }
    __syncthreads();
    if (t < 5 * S) {
      const int s = t / 5, c3 = t % 5;
      float a[1][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[0][e] = sm[O_B + 128 + 4 * c3 + e];
      product<64, 20, HS, 1>(sm + O_W3T, sm + Sh::O_H2, c3, s, a);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float d = b0 + s < n ? a[0][e] - __ldg(Y + int64_t(b0 + s) * D::NOUT + 4 * c3 + e) : 0.0f;
        lsum = fmaf(d, d, lsum);
        sm[Sh::O_DO + s * 20 + 4 * c3 + e] = 2.0f * d * inv_batch;
      }
    }
    __syncthreads();
    // ---- backward: dLoss/da2, then dLoss/da1 (in place of the derivatives)
    {
      float a[SPT][4] = {};
      product<20, 64, 20, SPT>(sm + O_W3, sm + Sh::O_DO, col, s0, a);
#pragma unroll
      for (int q = 0; q < SPT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) sm[Sh::O_D2 + (s0 + 16 * q) * HS + 4 * col + e] *= a[q][e];
    }
    __syncthreads();
    {
      float a[SPT][4] = {};
      product<64, 64, HS, SPT>(sm + O_W2, sm + Sh::O_D2, col, s0, a);
#pragma unroll
      for (int q = 0; q < SPT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) sm[Sh::O_D1 + (s0 + 16 * q) * HS + 4 * col + e] *= a[q][e];
    }
    __syncthreads();
    // ---- weight gradients of the tile, into registers
#pragma unroll 4
    for (int s = 0; s < S; ++s) {
      const float4 d1 = *reinterpret_cast<const float4*>(sm + Sh::O_D1 + s * HS + 4 * gr);
      const float2 x = *reinterpret_cast<const float2*>(sm + Sh::O_X + s * XS + 2 * gc);
      const float4 d2 = *reinterpret_cast<const float4*>(sm + Sh::O_D2 + s * HS + 4 * gr);
      const float4 h1 = *reinterpret_cast<const float4*>(sm + Sh::O_H1 + s * HS + 4 * gc);
      const float d1v[4] = {d1.x, d1.y, d1.z, d1.w}, d2v[4] = {d2.x, d2.y, d2.z, d2.w};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        g1[r][0] = fmaf(d1v[r], x.x, g1[r][0]);
        g1[r][1] = fmaf(d1v[r], x.y, g1[r][1]);
        fma4(g2[r], h1, d2v[r]);
      }
      const float h2 = sm[Sh::O_H2 + s * HS + (t & 63)];
#pragma unroll
      for (int r = 0; r < 5; ++r) g3[r] = fmaf(sm[Sh::O_DO + s * 20 + 5 * (t >> 6) + r], h2, g3[r]);
      if (t < 148)
        gb += t < 64 ? sm[Sh::O_D1 + s * HS + t] : t < 128 ? sm[Sh::O_D2 + s * HS + t - 64] : sm[Sh::O_DO + s * 20 + t - 128];
    }
  }
  // ---- the CTA's sums, through shared memory so that the additions are coalesced
  __syncthreads();
  float* row = sm;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (2 * gc + c < D::NIN) row[D::OFF_W1 + (4 * gr + r) * D::NIN + 2 * gc + c] = g1[r][c];
#pragma unroll
    for (int c = 0; c < 4; ++c) row[D::OFF_W2 + (4 * gr + r) * 64 + 4 * gc + c] = g2[r][c];
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) row[D::OFF_W3 + (5 * (t >> 6) + r) * 64 + (t & 63)] = g3[r];
  if (t < 148) row[t < 64 ? D::OFF_B1 + t : t < 128 ? D::OFF_B2 + t - 64 : D::OFF_B3 + t - 128] = gb;
  static_assert(O_ACT >= D::NPARAM, "the sums overlay the weights");
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if ((t & 31) == 0) atomicAdd(loss, double(lsum) * double(inv_batch));
  __syncthreads();
  // every CTA begins elsewhere, so that they do not queue at the same addresses
  constexpr int CH = (D::NPARAM + THREADS - 1) / THREADS;
  for (int k = 0; k < CH; ++k) {
    const int i = int((blockIdx.x + k) % CH) * THREADS + t;
    if (i < D::NPARAM) atomicAdd(sums + i, double(row[i]));
  }
}

// grad = sums, rounded; the loss behind them to *loss (pinned host memory; may be null)
__global__ void mlp_grad_round_kernel(const double* sums, float* grad, double* loss) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < MLPDims::NPARAM) grad[i] = float(sums[i]);
  else if (i == MLPDims::NPARAM && loss) *loss = sums[i];
}

}  // namespace sfem
