// DG SIPG Laplace (+ mass) in one launch for P3 (sm_100a).
//
// The operator is that of kernels_dg.cuh.  A P3 cell's normal derivatives on its
// faces cost too much to form once per side (89 operations a face), so a CTA
// publishes its cells' derivatives to itself, in shared memory, and forms those of
// the neighbours outside it from their values:
//   0. geometry by blocks, the CTA's rows, the rows of its outer neighbours and
//      the list of its outer faces come in with cp.async, all together;
//   1. a thread per cell and component forms the gradient, w = G grad u (which are
//      the derivatives on the faces up to sign and one sum), puts the face values
//      of w into shared memory and keeps h = MQ w; the outer faces' derivatives
//      are formed by as many threads as there are outer faces (64 to 128 cells of a
//      box in Morton order have 0.7 to 1 of them per cell);
//   2. the four faces from shared memory alone, then the transposed gradient.
// Against the two-launch form this saves the trace pass, its round trip (24 values
// a cell and component, written once and read twice) and the waits for
// neighbours in other CTAs, one per face.  B200, 45 x 38 x 31 hexes, us per vmult,
// two launches -> one: DG FP64 97 -> 66, FP32 55 -> 38; Helmholtz, 3 components,
// FP64 526 -> 231, FP32 252 -> 122.  FP64 32^3 by the profiler: 18.8 M warp
// instructions, FP64 pipe 36 %, issue slots 40 %, shared memory 47 %; 224 registers and
// 93 KB per CTA of 128 cells leave two of them an SM, 8 warps: bound by latency, 4.6
// cycles an instruction (the copies took 30 % of the cycles before the outer rows'
// indices were requested all at once, which took FP64 from 77 to 66 us).
#pragma once
#include <cstdint>

#include "kernels_dg_fused.cuh"

namespace sfem {

// Shared memory of a block: geometry (6 metric, 4 penalty, with mass 1 value per
// cell, then four 32-bit face codes), outer faces, rows, traces.
template <int NC, bool MASS, int BS, typename T>
struct Fused3Shape {
  using O = gen::Ops<3>;
  static constexpr int U = NC * O::K, US = U + 1;  // odd rows: a warp reads a node of its cells without conflicts
  static constexpr int NG = 10 + (MASS ? 1 : 0);
  static constexpr int GEO = NG * BS * int(sizeof(T)) + 4 * BS * 4;
  static constexpr int TR = 4 * O::NFQ;            // traces of a cell and component
  static constexpr int THREADS = BS * NC;
  static_assert(GEO % 16 == 0, "blocks of whole 16-byte units");
  // ne outer cells, nf outer faces
  static __host__ __device__ size_t bytes(int ne, int nf) {
    return GEO + size_t(nf) * 4 * sizeof(T) + size_t(ne) * 4 + (size_t(BS + ne) * US + size_t(TR) * THREADS + size_t(O::NFQ) * NC * nf) * sizeof(T);
  }
};
// face code: staged row | neighbour's face << 14 | outer face << 16; boundary: all ones
constexpr uint32_t kBoundary3 = 0xFFFFFFFFu;
// outer face: weights of its face vertices (J^-1 2|F| n, barycentric), then row | face << 14
template <typename T>
struct alignas(16) OuterFace {
  T w[3];
  union {
    T pad;
    uint32_t code;
  };
};

// byte offsets of side nodes 4 W .. 4 W + 3 of face F, one per byte
template <int F, typename T, int W>
__host__ __device__ constexpr uint32_t side3_word() {
  using O = gen::Ops<3>;
  return uint32_t(O::side(F, 4 * W) * sizeof(T)) | uint32_t(O::side(F, 4 * W + 1) * sizeof(T)) << 8 |
         uint32_t(O::side(F, 4 * W + 2) * sizeof(T)) << 16 | uint32_t(O::side(F, 4 * W + 3) * sizeof(T)) << 24;
}
// the first N values of a staged row in side order of its face f
template <int N, typename T, int W = 0>
__device__ __forceinline__ void row_side3(int f, const T* row, T (&s)[N]) {
  constexpr uint32_t w0 = side3_word<0, T, W>(), w1 = side3_word<1, T, W>(), w2 = side3_word<2, T, W>(),
                     w3 = side3_word<3, T, W>();
  const uint32_t lo = (f & 1) ? w1 : w0, hi = (f & 1) ? w3 : w2;
  const uint32_t w = (f & 2) ? hi : lo;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (4 * W + i < N)
      s[4 * W + i] = *reinterpret_cast<const T*>(reinterpret_cast<const unsigned char*>(row) + __byte_perm(w, 0, 0x4440 | i));
  if constexpr (4 * W + 4 < N) row_side3<N, T, W + 1>(f, row, s);
}

// Cells per CTA and resident CTAs that the registers are capped for.  Scalar, 45 x
// 38 x 31, us: FP64 128 cells 66.0, 64 66.3, 32 68.3 (five CTAs of 64 with 168
// registers and 108 bytes of spills: 5 % more); FP32 128 cells 38.1, 64 39.7, 32
// 43.0.  3 components: FP64 three CTAs 231, two 258; FP32 six 122, five 127, four 129;
// 64 cells would not hold the worst case, four outer neighbours each.
template <int NC>
__host__ __device__ constexpr int dg_fused3_cells() {
  return NC == 1 ? 128 : 32;
}
template <int NC, typename T>
__host__ __device__ constexpr int dg_fused3_min_ctas() {
  return sizeof(T) == 8 ? (NC == 1 ? 2 : 3) : (NC == 1 ? 4 : 6);
}

template <int NC, bool MASS, int BS, typename T, int MINB>
__global__ void __launch_bounds__(BS* NC, MINB)
    dg_fused3_kernel(const __grid_constant__ DGBatch<T> batch, int ne_max, int nf_max) {
  using O = gen::Ops<3>;
  using S = Fused3Shape<NC, MASS, BS, T>;
  constexpr int K = O::K, KQ = O::KQ, NF = O::NF, NFQ = O::NFQ, THREADS = S::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t blk = blockIdx.x;
  const int pi = find_problem(batch, blk);
  const DGProblem<T>& pr = batch.p[pi];
  const int64_t lb = blk - batch.block_begin[pi];
  const int64_t c0 = lb * BS;
  const int nloc = int(pr.n_cells - c0 < BS ? pr.n_cells - c0 : int64_t(BS));
  const int t = threadIdx.x, cell = t % BS, comp = t / BS;
  OuterFace<T>* sof = reinterpret_cast<OuterFace<T>*>(smem_raw + S::GEO);  // [nf_max]
  T* su = reinterpret_cast<T*>(sof + nf_max);                              // [BS + ne_max][US] rows, then results
  T* tq = su + (BS + ne_max) * S::US;                                      // [TR][THREADS] own traces
  T* tx = tq + S::TR * THREADS;                                            // [NFQ][NC nf_max] outer faces' traces
  int32_t* sx = reinterpret_cast<int32_t*>(tx + O::NFQ * NC * nf_max);     // [ne_max] outer neighbours
  // ---- 0: everything into shared memory
  const int32_t e0 = __ldg(pr.ext_begin + lb), ne = __ldg(pr.ext_begin + lb + 1) - e0;
  const int32_t f0 = __ldg(pr.face_begin + lb), nf = __ldg(pr.face_begin + lb + 1) - f0;
  OuterRows<BS, THREADS> outer;
  outer.load(pr.ext + e0, ne);
  {
    const unsigned char* g = pr.fgeo + lb * S::GEO;
    for (int e = t; e < S::GEO / 16; e += THREADS) cp_async_bytes<16>(smem_raw + 16 * e, g + 16 * e);
    const unsigned char* of = reinterpret_cast<const unsigned char*>(pr.outer) + size_t(f0) * sizeof(OuterFace<T>);
    for (int e = t; e < nf * int(sizeof(OuterFace<T>) / 16); e += THREADS)
      cp_async_bytes<16>(reinterpret_cast<unsigned char*>(sof) + 16 * e, of + 16 * e);
  }
  pdl_enter();  // the vectors' producer
  for (int e = t; e < nloc * S::U; e += THREADS)
    cp_async_bytes<sizeof(T)>(su + (e / S::U) * S::US + e % S::U, pr.src + c0 * S::U + e);
  outer.publish(sx, ne);
#pragma unroll 4
  for (int e = t; e < ne * S::U; e += THREADS) {
    const int r = e / S::U, v = e % S::U;
    cp_async_bytes<sizeof(T)>(su + (BS + r) * S::US + v, pr.src + int64_t(sx[r]) * S::U + v);
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  // ---- 1: own gradient and traces, outer faces' traces
  const T* sg = reinterpret_cast<const T*>(smem_raw) + cell;
  const uint32_t* sc = reinterpret_cast<const uint32_t*>(smem_raw + S::NG * BS * sizeof(T)) + cell;
  T* own = su + cell * S::US + comp * K;
  T h[3 * KQ];
  if (cell < nloc) {
    T u[K], g[3 * KQ], w[3 * KQ], G[6];
#pragma unroll
    for (int i = 0; i < K; ++i) u[i] = own[i];
#pragma unroll
    for (int k = 0; k < 6; ++k) G[k] = sg[k * BS];
    O::grad(u, g);
    apply_metric<KQ>(G, g, w);
#pragma unroll
    for (int m = 0; m < NFQ; ++m) {
      const int n0 = O::fnq(0, m);
      tq[m * THREADS + t] = w[n0] + w[KQ + n0] + w[2 * KQ + n0];
#pragma unroll
      for (int f = 1; f < 4; ++f) tq[(f * NFQ + m) * THREADS + t] = -w[(f - 1) * KQ + O::fnq(f, m)];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) O::massQ(w + a * KQ, h + a * KQ);
  }
  for (int e = t; e < nf * NC; e += THREADS) {
    const int k = e % nf, cp = e / nf;
    const OuterFace<T> of = sof[k];
    T s[K], d[3 * NFQ];
    row_side3<K>(int(of.code >> 14 & 3u), su + (of.code & 0x3FFFu) * S::US + cp * K, s);
    O::sideGrad(s, d);
#pragma unroll
    for (int m = 0; m < NFQ; ++m)
      tx[m * (NC * nf_max) + cp * nf_max + k] = of.w[0] * d[m] + of.w[1] * d[NFQ + m] + of.w[2] * d[2 * NFQ + m];
  }
  __syncthreads();
  // ---- 2: faces, transposed gradient
  T y[K];
  if (cell < nloc) {
#pragma unroll
    for (int i = 0; i < K; ++i) y[i] = T(0);
    if (MASS) {
      T u[K];
#pragma unroll
      for (int i = 0; i < K; ++i) u[i] = own[i];
      O::massP(u, sg[10 * BS], y);
    }
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const uint32_t code = sc[f * BS];
      T j[NF], dq[NFQ];
      if (code != kBoundary3) {
        const int row = int(code & 0x3FFFu), nbf = int(code >> 14 & 3u);
        row_side3<NF>(nbf, su + row * S::US + comp * K, j);
#pragma unroll
        for (int i = 0; i < NF; ++i) j[i] = own[O::fn(f, i)] - j[i];
        const bool in = row < BS;
        const T* qn = in ? tq + nbf * NFQ * THREADS + comp * BS + row : tx + comp * nf_max + (code >> 16);
        const int qs = in ? THREADS : NC * nf_max;
#pragma unroll
        for (int m = 0; m < NFQ; ++m) dq[m] = tq[(f * NFQ + m) * THREADS + t] - qn[m * qs];
      } else {
        // u+ = -u-, d_n u+ = d_n u-
#pragma unroll
        for (int i = 0; i < NF; ++i) j[i] = T(2) * own[O::fn(f, i)];
#pragma unroll
        for (int m = 0; m < NFQ; ++m) dq[m] = T(2) * tq[(f * NFQ + m) * THREADS + t];
      }
      T G[6], cf[3];
#pragma unroll
      for (int k = 0; k < 6; ++k) G[k] = sg[k * BS];
      face_cf(G, f, cf);
      face_apply<3>(f, j, dq, sg[(6 + f) * BS], cf, h, y);
    }
    O::gradT(h, y);
  }
  __syncthreads();  // every thread is done with the staged rows
  if (cell < nloc) {
#pragma unroll
    for (int i = 0; i < K; ++i) own[i] = y[i];
  }
  __syncthreads();
  copy_rows_out<S::U, S::US, BS, THREADS>(pr.dst + c0 * S::U, su, nloc);
}

}  // namespace sfem
