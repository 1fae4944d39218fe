// Continuous Galerkin Laplace on Kuhn boxes: one thread per hex, 4 x 4 x 4 hexes
// per CTA step (sm_100a).
//
// The operator is that of kernels_cg.cuh.  A block of 4 x 4 x 4 hexes has
// (4 P + 1)^3 lattice nodes, and a hex's nodes sit at fixed offsets from its
// corner, so nothing about the block's connectivity is read from tables:
//   1. the block's DoF values are gathered once into a lattice array in shared
//      memory (cp.async, one block ahead);
//   2. every thread takes its hex's (P + 1)^3 values into registers, applies the
//      six tet operators (compile-time node numbers) and adds them up in
//      registers;
//   3. the hexes' results are added into a second lattice array without atomics:
//      for a fixed node offset the 64 hexes write 64 different nodes, and offsets
//      that can meet (the lower sides of a hex and the upper sides of its
//      neighbour) are taken in eight phases, ordered by warp barriers and, where
//      the two warps meet, one CTA barrier;
//   4. every lattice node is written back once: a store where no other block
//      touches the DoF, else an atomic.
// The thread-per-tet cube kernel reads and writes every tet's nodes through
// shared memory (P2: 60 reads, 60 writes, 60 reduction reads per hex and their
// index tables) and is bound by that; here it is 27 reads and 46 accesses for the
// sums, all without bank conflicts (the lattice is stored with x split by residue
// mod P and row / plane strides chosen for it).
// Blocks at the sides of a box whose sides 4 does not divide are padded: absent
// hexes have a zero metric, absent nodes the code of constrained DoFs.
//
// Measured on B200 against the thread-per-tet forms, back to back: P2 FP64 128^3
// 343 -> 272 us, FP32 252 -> 155 us; P1 FP64 128^3 139 -> 101 us (the metric
// alone is 92 us of HBM), FP32 74.5 -> 54 us; P3 FP32 64^3 100.6 -> 89.5 us; P2
// FP64 on 37 x 41 x 35 hexes 18.7 -> 13.5 us.  What is left for P2 FP64 (128^3, by the
// profiler) is latency: 12 warps per SM of 168 registers, 8.5 cycles an instruction;
// FP64 pipe 35 %, L1 and shared memory 61 %, HBM 52 % busy (62 % of the bytes that the
// kernel needs are the stored metric).  P3 FP32 64^3: 8 warps of 222 registers, 5.0
// cycles, issue slots 40 %, L1 and shared memory 33 %.  Where the form is the default:
// CGBlocks::pays.
//
// codes [n_blocks][NBP] DoF | interior << 30, -1: constrained or absent node
// pos   [NBP]           lattice position of slot n (the same for every block;
//                       see cg_block_slots)
// geo   [n_blocks][36][64] metric value k of tet q of hex t at [6 q + k][t]
#pragma once
#include <cstdint>

#include "kernels_cg.cuh"

namespace sfem {

template <int P, typename T>
struct CGBlockShape {
  static constexpr int N1 = 4 * P + 1, NB = N1 * N1 * N1, H1 = P + 1, H = H1 * H1 * H1;
  static constexpr int NBP = (NB + 63) / 64 * 64;
  // row and plane strides (values).  A warp's hexes are 4 x 4 x 2; their accesses
  // at one offset start at hx + P SY hy + P SZ hz: 16 lanes of 8-byte values
  // (one wavefront) need P SY = 4 or 12 mod 16, 32 lanes of 4-byte values
  // P SY = 4, 12, 20 or 28 and P SZ = 16 mod 32.
  static constexpr int SY = P == 1 ? 12 : P == 2 ? 10 : 20;
  static constexpr int SZ = sizeof(T) == 8 ? N1 * SY : P == 1 ? 80 : P == 2 ? 104 : 272;
  static_assert(SY >= N1 && SZ >= (N1 - 1) * SY + N1, "lattice strides");
  static_assert(sizeof(T) == 8 ? (P * SY) % 8 == 4 : (P * SY) % 8 == 4 && (P * SZ) % 32 == 16, "bank pattern");
  static constexpr int LAT = (N1 - 1) * (SZ + SY) + N1;  // then one slot for the padding entries
  static constexpr int LATP = (LAT + 1 + 3) / 4 * 4;
  // position of lattice node (x, y, z): x split by residue mod P
  static __host__ __device__ constexpr int xpos(int x) { return x % P == 0 ? x / P : 5 + 4 * (x % P - 1) + x / P; }
  static __host__ __device__ constexpr int at(int x, int y, int z) { return xpos(x) + SY * y + SZ * z; }
  // offset of hex node (a, b, c) from the hex's base hx + P SY hy + P SZ hz
  static __host__ __device__ constexpr int off(int a, int b, int c) {
    return (a == 0 ? 0 : a == P ? 1 : 5 + 4 * (a - 1)) + SY * b + SZ * c;
  }
  // code ring: with three slots the codes come in two blocks ahead; P3 has two (a
  // third would cost a resident CTA: P3 FP32 64^3 116 us instead of 89, while P2
  // FP64 128^3 takes 285 us with two slots)
  static constexpr int RING = P <= 2 ? 3 : 2;
  static constexpr int PRE = RING * NBP * 4 + NBP * 2;  // codes, positions
  static constexpr size_t bytes(int nc) { return PRE + size_t(2) * nc * LATP * sizeof(T); }
  static_assert(PRE % 16 == 0, "value arrays start aligned");
};

// y(i) += (A_K u)_i
template <int P, typename T, class F>
__device__ __forceinline__ void cg_local_apply_into(const T (&G)[6], const T (&u)[gen::Ops<P>::K], F&& y) {
  using O = gen::Ops<P>;
  T g[3 * O::KQ], w[3 * O::KQ];
  O::grad(u, g);
  apply_metric<O::KQ>(G, g, w);
#pragma unroll
  for (int a = 0; a < 3; ++a) O::massQ(w + a * O::KQ, g + a * O::KQ);
  O::gradTInto(g, y);
}

template <int P, typename T, int NC, int MINB>
__global__ void __launch_bounds__(64, MINB)
    cg_block_kernel(int64_t n_blocks, const int32_t* __restrict__ codes, const int16_t* __restrict__ pos,
                    const T* __restrict__ geo, const T* __restrict__ src, T* __restrict__ dst, int64_t n_constrained,
                    const int32_t* __restrict__ constrained) {
  using S = CGBlockShape<P, T>;
  using O = gen::Ops<P>;
  constexpr int NBP = S::NBP, H1 = S::H1;
  extern __shared__ __align__(16) unsigned char smem_blk[];
  int32_t* ring = reinterpret_cast<int32_t*>(smem_blk);        // [RING][NBP]
  int16_t* sp = reinterpret_cast<int16_t*>(ring + S::RING * NBP);    // [NBP]
  T* ub = reinterpret_cast<T*>(smem_blk + S::PRE);             // [NC][LATP] gathered values
  T* yb = ub + NC * S::LATP;                                   // [NC][LATP] sums
  const int t = threadIdx.x;
  const int64_t stride = gridDim.x;
  for (int e = t; e < NBP / 8; e += 64)
    reinterpret_cast<uint4*>(sp)[e] = __ldg(reinterpret_cast<const uint4*>(pos) + e);
  auto issue_codes = [&](int64_t b, int slot) {
    if (b < n_blocks)
      for (int e = t; e < NBP / 4; e += 64) {
        const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(ring + slot * NBP + 4 * e));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(codes + b * NBP + 4 * e) : "memory");
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto issue_gather = [&](int64_t b, int slot) {
    if (b < n_blocks) {
#pragma unroll 4
      for (int q = 0; q < NBP / 64; ++q) {
        const int n = t + 64 * q;
        const int32_t c = ring[slot * NBP + n];
        T* d = ub + sp[n];
#pragma unroll
        for (int k = 0; k < NC; ++k) {
          if (c < 0) {
            d[k * S::LATP] = T(0);
          } else {
            const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(d + k * S::LATP));
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(sa),
                         "l"(src + int64_t(NC) * (c & 0x3FFFFFFF) + k), "n"(sizeof(T))
                         : "memory");
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int hx = t & 3, hy = (t >> 2) & 3, hz = t >> 4;
  const int base = hx + P * S::SY * hy + P * S::SZ * hz;
  // metric of tet q of this thread's hex in block b (q = 6: tet 0 of the next block)
  auto load_geo = [&](int64_t b, int q, T (&G)[6]) {
    const T* p = geo + ((b + (q == 6 ? stride : 0)) * 36 + (q == 6 ? 0 : 6 * q)) * 64 + t;
    const bool in = q < 6 || b + stride < n_blocks;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      G[k] = T(0);
      if (in) G[k] = ld_stream(p + 64 * k);
    }
  };

  int64_t b = blockIdx.x;
  issue_codes(b, 0);
  T G[2][6];
  if (b < n_blocks) load_geo(b, 0, G[0]);
  pdl_enter();  // the operator's own tables are on their way; src and dst from here on
  for (int64_t i = blockIdx.x * int64_t(64) + t; i < n_constrained; i += stride * 64) {
    const int32_t g = constrained[i];
    dst[g] = src[g];
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  issue_gather(b, 0);
  issue_codes(b + stride, 1);
  int cur = 0;  // ring slot of block b's codes
  for (; b < n_blocks; b += stride) {
    const int nxt = cur + 1 == S::RING ? 0 : cur + 1;
    asm volatile("cp.async.wait_group 0;" ::: "memory");  // this block's values, the next one's codes
    __syncthreads();
    if (S::RING == 3) issue_codes(b + 2 * stride, nxt + 1 == 3 ? 0 : nxt + 1);
#pragma unroll 1
    for (int k = 0; k < NC; ++k) {
      const T* uk = ub + k * S::LATP + base;
      T* yk = yb + k * S::LATP + base;
      T u[S::H], y[S::H];
#pragma unroll
      for (int c = 0; c < H1; ++c)
#pragma unroll
        for (int bb = 0; bb < H1; ++bb)
#pragma unroll
          for (int a = 0; a < H1; ++a) {
            u[a + H1 * (bb + H1 * c)] = uk[S::off(a, bb, c)];
            y[a + H1 * (bb + H1 * c)] = T(0);
          }
      if (k == NC - 1) {
        __syncthreads();  // every thread has its values: the next block's may come in
        issue_gather(b + stride, nxt);
      }
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        // the next tet's metric is requested before this one's arithmetic
        if (NC == 1 || k == NC - 1 || q < 5) load_geo(b, q + 1, G[(q + 1) & 1]);
        else load_geo(b, 0, G[(q + 1) & 1]);
        T ut[O::K];
#pragma unroll
        for (int i = 0; i < O::K; ++i) ut[i] = u[O::hex_node(q, i)];
        cg_local_apply_into<P>(G[q & 1], ut, [&](int i) -> T& { return y[O::hex_node(q, i)]; });
      }
      // sums over the hexes: lower sides first, then upper sides onto the
      // neighbours' lower ones, z outermost (only its upper side meets the other warp)
#pragma unroll
      for (int ph = 0; ph < 8; ++ph) {
        const int A = ph & 1, B = (ph >> 1) & 1, C = ph >> 2;
        if (ph == 4) __syncthreads();
        else if (ph > 0) __syncwarp();
        // a node of an upper side has a sum already unless the block ends there
        const bool has = (A && hx < 3) || (B && hy < 3) || (C && hz < 3);
#pragma unroll
        for (int c = C ? P : 0; c < (C ? P + 1 : P); ++c)
#pragma unroll
          for (int bb = B ? P : 0; bb < (B ? P + 1 : P); ++bb)
#pragma unroll
            for (int a = A ? P : 0; a < (A ? P + 1 : P); ++a) {
              T* d = yk + S::off(a, bb, c);
              const T v = y[a + H1 * (bb + H1 * c)];
              if (ph == 0) *d = v;
              else *d = has ? *d + v : v;
            }
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int q = 0; q < NBP / 64; ++q) {
      const int n = t + 64 * q;
      const int32_t c = ring[cur * NBP + n];
      if (c < 0) continue;
      const T* v = yb + sp[n];
      T* d = dst + int64_t(NC) * (c & 0x3FFFFFFF);
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        if (c & 0x40000000) d[k] = v[k * S::LATP];
        else atomicAdd(d + k, v[k * S::LATP]);
      }
    }
    if (S::RING == 2) {
      __syncthreads();  // every thread is done with this block's codes
      issue_codes(b + 2 * stride, cur);
    }
    cur = nxt;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace sfem
