// DG SIPG Laplace (+ mass) in one pass for P1 and P2 (sm_100a).
//
// The operator is that of kernels_dg.cuh.  There, a first pass publishes every
// cell's normal derivatives on its faces and the second reads the neighbours';
// for P1 and P2 it is cheaper to form the neighbour's derivative where it is
// needed.  With c_w = J^-1 (2|F| n) as barycentric weights (c_0 = -c_1 - c_2 -
// c_3, they add up to zero) the scaled normal derivative is
//   P1:  q   = sum_w c_w u_w                        (constant on the face)
//   P2:  q_v = 4 sum_w c_w u_vw - sum_w c_w u_w     at face vertex v, u_vw the
//              value at the midpoint of edge vw and u_vv = u_v,
// 4 and 19 multiply-adds for a face, from the neighbour's values (which the jump
// reads in part anyway) and three numbers c^+ of the neighbour's geometry per
// face.  The published traces are 12 and 36 values per cell for three components
// (written once, read twice).
//
// One thread per cell and component: a warp's 32 cells are contiguous and have
// one component.  A CTA has BS cells; their rows and the rows of every neighbour
// outside the CTA (a list made at set-up, each cell once) are copied into shared
// memory with cp.async, all in flight together, so that the faces read shared
// memory only: a neighbour's row costs 240 contiguous bytes (P2, three
// components) instead of 30 scattered 8-byte loads in as many divergent
// branches.  On a box in Morton order 64 cells have about 60 such neighbours.
// The nodes of a neighbour's face are addressed by byte offsets picked from four
// packed constants by the neighbour's face number, without branches.
//
// The geometry is stored by blocks of cells and copied with the rows, so that
// nothing is waited for after the one staging (loading it face by face instead:
// P2 FP64, three components 117 us, neighbours from global memory too 115 us,
// staged 80 us).  The faces come first, then the cell term, which keeps the live
// values to about 50.  What is left by the profiler (cold caches) for P2 FP64, three
// components: shared-memory wavefronts 69 %, issue slots 49 %, FP64 pipe 42 % busy; for
// scalar P2 FP32 the issue slots (65 %).  Persistent CTAs that copy the next block during the arithmetic were not
// faster (105 us: the second stage costs resident warps).
#pragma once
#include <cstdint>

#include "kernels_dg.cuh"

namespace sfem {

// A cell's values from the side of face F: face nodes in canonical order, then
// the other values its normal derivative needs.  P1: three face vertices, the
// opposite vertex.  P2: the six face nodes (v0 m01 m02 v1 m12 v2), the opposite
// vertex o, the midpoints o-v0, o-v1, o-v2.
template <int P, int F, int I>
__host__ __device__ constexpr int side_node() {
  // edge number of local vertices a < b
  constexpr int E[4][4] = {{0, 4, 5, 6}, {4, 0, 7, 8}, {5, 7, 0, 9}, {6, 8, 9, 0}};
  constexpr int v[3] = {F == 0 ? 1 : 0, F <= 1 ? 2 : 1, F <= 2 ? 3 : 2};
  if (P == 1) return I < 3 ? v[I < 3 ? I : 0] : F;
  constexpr int face[6] = {v[0], E[v[0]][v[1]], E[v[0]][v[2]], v[1], E[v[1]][v[2]], v[2]};
  if (I < 6) return face[I < 6 ? I : 0];
  if (I == 6) return F;
  return E[F][v[I >= 7 && I < 10 ? I - 7 : 0]];
}

template <int P, int F, typename T, int I = 0>
__device__ __forceinline__ void own_side(const T (&u)[gen::Ops<P>::K], T (&s)[gen::Ops<P>::K]) {
  s[I] = u[side_node<P, F, I>()];  // a renaming of registers
  if constexpr (I + 1 < gen::Ops<P>::K) own_side<P, F, T, I + 1>(u, s);
}
// byte offsets of side nodes 4 W .. 4 W + 3 of face F, one per byte
template <int P, int F, typename T, int W, int I = 0>
__host__ __device__ constexpr uint32_t side_word() {
  constexpr int k = 4 * W + I;
  constexpr uint32_t v = k < gen::Ops<P>::K ? uint32_t(side_node<P, F, (k < gen::Ops<P>::K ? k : 0)>() * sizeof(T)) << (8 * I) : 0u;
  if constexpr (I < 3) return v | side_word<P, F, T, W, I + 1>();
  else return v;
}
// the values of a staged row in side order of its face f (known at run time)
template <int P, typename T, int W = 0>
__device__ __forceinline__ void row_side(int f, const T* row, T (&s)[gen::Ops<P>::K]) {
  constexpr int K = gen::Ops<P>::K;
  const uint32_t lo = (f & 1) ? side_word<P, 1, T, W>() : side_word<P, 0, T, W>();
  const uint32_t hi = (f & 1) ? side_word<P, 3, T, W>() : side_word<P, 2, T, W>();
  const uint32_t w = (f & 2) ? hi : lo;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (4 * W + i < K)
      s[4 * W + i] = *reinterpret_cast<const T*>(reinterpret_cast<const unsigned char*>(row) + __byte_perm(w, 0, 0x4440 | i));
  if constexpr (4 * W + 4 < K) row_side<P, T, W + 1>(f, row, s);
}

// weights c in side order (three face vertices, opposite vertex) from J^-1 (2|F| n)
template <int F, typename T>
__device__ __forceinline__ void side_weights(const T (&cf)[3], T (&c)[4]) {
  const T c0 = -(cf[0] + cf[1] + cf[2]);
  const T w[4] = {c0, cf[0], cf[1], cf[2]};
  c[0] = w[F == 0 ? 1 : 0];
  c[1] = w[F <= 1 ? 2 : 1];
  c[2] = w[F <= 2 ? 3 : 2];
  c[3] = w[F];
}

// difference of the two sides' scaled outward normal derivatives at the P_{p-1} face nodes
template <int P, typename T>
__device__ __forceinline__ void side_flux(const T (&c)[4], const T (&s)[gen::Ops<P>::K], const T (&cn)[4],
                                          const T (&sn)[gen::Ops<P>::K], T (&dq)[gen::Ops<P>::NFQ]) {
  if constexpr (P == 1) {
    T a = c[0] * s[0];
#pragma unroll
    for (int w = 1; w < 4; ++w) a += c[w] * s[w];
#pragma unroll
    for (int w = 0; w < 4; ++w) a -= cn[w] * sn[w];
    dq[0] = a;
  } else {
    // vertices in side order: s[0], s[3], s[5], s[6]; midpoint of side vertices (i, j)
    constexpr int V[4] = {0, 3, 5, 6};
    constexpr int M[3][4] = {{0, 1, 2, 7}, {1, 3, 4, 8}, {2, 4, 5, 9}};
    T ds = c[0] * s[V[0]];
#pragma unroll
    for (int w = 1; w < 4; ++w) ds += c[w] * s[V[w]];
#pragma unroll
    for (int w = 0; w < 4; ++w) ds -= cn[w] * sn[V[w]];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      T a = c[0] * s[M[v][0]];
#pragma unroll
      for (int w = 1; w < 4; ++w) a += c[w] * s[M[v][w]];
#pragma unroll
      for (int w = 0; w < 4; ++w) a -= cn[w] * sn[M[v][w]];
      dq[v] = T(4) * a - ds;
    }
  }
}

// Staged rows: U = NC K values, padded so that a row is an odd number of vectors
// of two values; a thread's own row is then read and written by vectors without
// bank conflicts, and copied by 16 (FP64) or 8 (FP32) bytes at a time.
template <int P, int NC, bool MASS, int BS, typename T>
struct FusedShape {
  static constexpr int U = NC * gen::Ops<P>::K;
  static_assert(U % 2 == 0, "rows of whole vectors");
  static constexpr int US = (U / 2) % 2 ? U : U + 2;
  static constexpr int CB = 2 * int(sizeof(T));  // bytes of a vector
  static constexpr int CH = U / 2;               // vectors of a row
  // geometry of a block: 6 metric, 4 penalty, 12 neighbour weights and (mass) 1
  // values per cell, then the four face codes
  static constexpr int NG = 22 + (MASS ? 1 : 0);
  static constexpr int GEO = NG * BS * int(sizeof(T)) + 4 * BS * 2;  // bytes, a multiple of 16
  static_assert(GEO % 16 == 0, "blocks of whole 16-byte units");
  static __host__ __device__ size_t bytes(int rows) { return GEO + size_t(rows) * US * sizeof(T) + size_t(rows - BS) * 4; }
};
template <typename T>
struct alignas(2 * sizeof(T)) Vec2 {
  T x, y;
};

template <int CB>
__device__ __forceinline__ void cp_async_bytes(void* smem, const void* gmem) {
  const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  if constexpr (CB == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(sa), "l"(gmem), "n"(CB) : "memory");
}

// code of a cell's face (in the block's geometry): staged row << 2 | the neighbour's face number, kBoundary
// on a boundary face
constexpr uint16_t kBoundary = 0xFFFF;

template <int P, int NC, int BS, int F, typename T>
__device__ __forceinline__ void dg_fused_face(const T* sg, const uint16_t* sc, int comp, const T* su,
                                              const T (&u)[gen::Ops<P>::K], const T (&G)[6],
                                              T (&h)[3 * gen::Ops<P>::KQ], T (&y)[gen::Ops<P>::K]) {
  using O = gen::Ops<P>;
  using S = FusedShape<P, NC, false, BS, T>;
  constexpr int K = O::K, NF = O::NF, NFQ = O::NFQ;
  const uint32_t code = sc[F * BS];
  const T sf = sg[(6 + F) * BS];
  T cfn[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) cfn[a] = sg[(10 + 3 * F + a) * BS];
  T s[K], sn[K], cf[3], cw[4], cn[4];
  own_side<P, F>(u, s);
  face_cf(G, F, cf);
  side_weights<F>(cf, cw);
  if (code != kBoundary) {
    row_side<P>(int(code & 3u), su + (code >> 2) * S::US + comp * K, sn);
    cn[0] = cfn[0];
    cn[1] = cfn[1];
    cn[2] = cfn[2];
    cn[3] = -(cfn[0] + cfn[1] + cfn[2]);
  } else {
    // u+ = -u-, d_n u+ = d_n u-
#pragma unroll
    for (int i = 0; i < K; ++i) sn[i] = -s[i];
#pragma unroll
    for (int w = 0; w < 4; ++w) cn[w] = cw[w];
  }
  T dq[NFQ], j[NF];
  side_flux<P>(cw, s, cn, sn, dq);
#pragma unroll
  for (int i = 0; i < NF; ++i) j[i] = s[i] - sn[i];
  face_apply<P>(F, j, dq, sf, cf, h, y);
}

// Cells per CTA (128 threads for scalar problems, 192 for three components) and
// resident CTAs that the registers are capped for.  More resident warps won
// throughout until spills cost more: P2 FP64 three components 64 cells, three
// CTAs (96 registers) 86 us, two (164, no spills) 101, four 113 us; P2 FP32 five
// CTAs 50, four 56 us; P1 FP32 scalar twelve CTAs 9.1, eight 9.6 us (45 x 38 x 31
// hexes).
template <int NC>
__host__ __device__ constexpr int dg_fused_cells() {
  return NC == 1 ? 128 : 64;
}
template <int P, int NC, typename T>
__host__ __device__ constexpr int dg_fused_min_ctas() {
  return sizeof(T) == 8 ? (P == 1 ? (NC == 1 ? 8 : 5) : (NC == 1 ? 4 : 3)) : (P == 1 ? (NC == 1 ? 12 : 6) : (NC == 1 ? 8 : 5));
}

// Rows of the outer neighbours of a block (at most 4 per cell): every index is
// requested at once, ahead of the copies that need none of them, and goes
// through shared memory to the threads that copy the rows.  Against a load per
// copied value ahead of its copy (B200, 45 x 38 x 31 hexes): P2 FP64, three
// components 85.5 -> 79.5 us, P1 37.9 -> 32.6, scalar P2 27.8 -> 25.5, scalar P2 FP32
// 17.0 -> 16.2.  Padding the lists to one length, which saves the wait for their
// beginnings, gave another 1 %: not kept.
template <int BS, int THREADS>
struct OuterRows {
  static constexpr int N = (4 * BS + THREADS - 1) / THREADS;
  int32_t v[N];
  __device__ __forceinline__ void load(const int32_t* ext, int ne) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int r = int(threadIdx.x) + i * THREADS;
      v[i] = r < ne ? __ldg(ext + r) : 0;
    }
  }
  __device__ __forceinline__ void publish(int32_t* s, int ne) const {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int r = int(threadIdx.x) + i * THREADS;
      if (r < ne) s[r] = v[i];
    }
    __syncthreads();
  }
};

template <int P, int NC, bool MASS, int BS, typename T, int MINB>
__global__ void __launch_bounds__(BS* NC, MINB) dg_fused_kernel(const __grid_constant__ DGBatch<T> batch, int rows) {
  using O = gen::Ops<P>;
  using S = FusedShape<P, NC, MASS, BS, T>;
  constexpr int K = O::K, KQ = O::KQ, THREADS = BS * NC;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // geometry, then the rows of the CTA's cells (later the results) and of its outer neighbours
  T* su = reinterpret_cast<T*>(smem_raw + S::GEO);
  const int64_t blk = blockIdx.x;
  const int pi = find_problem(batch, blk);
  const DGProblem<T>& pr = batch.p[pi];
  const int64_t lb = blk - batch.block_begin[pi];
  const int64_t c0 = lb * BS;
  const int nloc = int(pr.n_cells - c0 < BS ? pr.n_cells - c0 : int64_t(BS));
  const int t = threadIdx.x, cell = t % BS, comp = t / BS;
  // ---- geometry and rows into shared memory
  const int32_t e0 = __ldg(pr.ext_begin + lb), ne = __ldg(pr.ext_begin + lb + 1) - e0;
  int32_t* sx = reinterpret_cast<int32_t*>(su + rows * S::US);  // [rows - BS] outer neighbours
  OuterRows<BS, THREADS> outer;
  outer.load(pr.ext + e0, ne);
  {
    const unsigned char* g = pr.fgeo + lb * S::GEO;
    for (int e = t; e < S::GEO / 16; e += THREADS) cp_async_bytes<16>(smem_raw + 16 * e, g + 16 * e);
  }
  pdl_enter();  // the vectors' producer
  if ((reinterpret_cast<uintptr_t>(pr.src) & uintptr_t(S::CB - 1)) == 0) {
    const T* own = pr.src + c0 * S::U;
    for (int e = t; e < nloc * S::CH; e += THREADS)
      cp_async_bytes<S::CB>(su + (e / S::CH) * S::US + 2 * (e % S::CH), own + 2 * e);
    outer.publish(sx, ne);
#pragma unroll 4
    for (int e = t; e < ne * S::CH; e += THREADS) {
      const int r = e / S::CH, v = e % S::CH;
      cp_async_bytes<S::CB>(su + (BS + r) * S::US + 2 * v, pr.src + int64_t(sx[r]) * S::U + 2 * v);
    }
  } else {
    for (int e = t; e < nloc * S::U; e += THREADS)
      cp_async_bytes<sizeof(T)>(su + (e / S::U) * S::US + e % S::U, pr.src + c0 * S::U + e);
    outer.publish(sx, ne);
    for (int e = t; e < ne * S::U; e += THREADS) {
      const int r = e / S::U, v = e % S::U;
      cp_async_bytes<sizeof(T)>(su + (BS + r) * S::US + v, pr.src + int64_t(sx[r]) * S::U + v);
    }
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  T* own = su + cell * S::US + comp * K;
  T y[K];
  if (cell < nloc) {
    const T* sg = reinterpret_cast<const T*>(smem_raw) + cell;
    const uint16_t* sc = reinterpret_cast<const uint16_t*>(smem_raw + S::NG * BS * sizeof(T)) + cell;
    T G[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) G[k] = sg[k * BS];
    T h[3 * KQ], u[K];
#pragma unroll
    for (int i = 0; i < K; i += 2) {
      const Vec2<T> v = *reinterpret_cast<const Vec2<T>*>(own + i);
      u[i] = v.x;
      u[i + 1] = v.y;
    }
#pragma unroll
    for (int i = 0; i < 3 * KQ; ++i) h[i] = T(0);
#pragma unroll
    for (int i = 0; i < K; ++i) y[i] = T(0);
    dg_fused_face<P, NC, BS, 0>(sg, sc, comp, su, u, G, h, y);
    dg_fused_face<P, NC, BS, 1>(sg, sc, comp, su, u, G, h, y);
    dg_fused_face<P, NC, BS, 2>(sg, sc, comp, su, u, G, h, y);
    dg_fused_face<P, NC, BS, 3>(sg, sc, comp, su, u, G, h, y);
    T g[3 * KQ], w[3 * KQ];
    O::grad(u, g);
    apply_metric<KQ>(G, g, w);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      T o[KQ];
      O::massQ(w + a * KQ, o);
#pragma unroll
      for (int m = 0; m < KQ; ++m) h[a * KQ + m] += o[m];
    }
    if (MASS) O::massP(u, sg[22 * BS], y);
    O::gradT(h, y);
  }
  // ---- results through the CTA's rows, stored coalesced
  __syncthreads();  // every thread is done with the staged rows
  if (cell < nloc) {
#pragma unroll
    for (int i = 0; i < K; i += 2) *reinterpret_cast<Vec2<T>*>(own + i) = Vec2<T>{y[i], y[i + 1]};
  }
  __syncthreads();
  T* out = pr.dst + c0 * S::U;
  if ((reinterpret_cast<uintptr_t>(pr.dst) & uintptr_t(S::CB - 1)) == 0) {
    for (int e = t; e < nloc * S::CH; e += THREADS)
      *reinterpret_cast<Vec2<T>*>(out + 2 * e) =
          *reinterpret_cast<const Vec2<T>*>(su + (e / S::CH) * S::US + 2 * (e % S::CH));
  } else {
    for (int e = t; e < nloc * S::U; e += THREADS) out[e] = su[(e / S::U) * S::US + e % S::U];
  }
}

}  // namespace sfem
