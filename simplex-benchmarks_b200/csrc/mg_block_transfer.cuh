// p-transfers of the multigrid (P_p <-> P_{p-1} on one Kuhn box) by blocks of 4 x 4
// x 4 hexes (the blocks and codes of kernels_cg_block.cuh).
//
// A fine node's value is interpolated from the coarse nodes of the edge or face it
// lies on (1, 2, 3 or 6 of them), and in the lattice of a block that rule is the
// same for every block: two small tables serve all of them.  A persistent CTA
// gathers a block's values into shared memory once, and every node is read and
// written once: the fine nodes by the block that owns them (a node on an upper
// side of the block belongs to the next block, if there is one), the coarse ones
// with an addition where no other block touches them and an atomic otherwise.
// The thread-per-cell forms gather every node from each of its cells through
// the 20-wide table; on 64^3 P3 <-> P2 (FP32, B200) they take 102 us
// (prolongation) and 128 us (restriction) for 70 MB.
//
// Arithmetic in FP64, as in the other forms.  MINUS forms the residual b - t on the
// way, which saves writing and reading it.
#pragma once
#include <cstdint>

#include "pdl.cuh"

namespace sfem {

struct BlockTransferTables {
  const uint16_t* ent;   // [6][NBPf] coarse slot | weight << 12 of a fine slot's entries
  const uint8_t* hi;     // [NBPf] bit d: the slot lies on the upper side in direction d
  const uint16_t* list;  // coarse slots' entries: fine slot | weight << 12
  const int32_t* start;  // [NBPc + 1]
  const uint16_t* order; // [NBPc] coarse slots, longest lists first
  int32_t n_list;
};
struct BlockWeights {
  double w[8];  // w[7] = 0
};

constexpr int kXferThreads = 256;

// xf += P xc
template <typename T, int NBPF, int NBPC>
__global__ void __launch_bounds__(kXferThreads)
    block_prolongate_add(int64_t n_blocks, const __grid_constant__ BlockTransferTables tb,
                         const __grid_constant__ BlockWeights wt, const uint8_t* __restrict__ upper,
                         const int32_t* __restrict__ fcodes, const int32_t* __restrict__ ccodes,
                         const T* xc, T* xf) {
  extern __shared__ __align__(16) unsigned char smem_x[];
  double* sw = reinterpret_cast<double*>(smem_x);                // [8]
  T* uc = reinterpret_cast<T*>(smem_x + 64);                     // [NBPC]
  uint16_t* ent = reinterpret_cast<uint16_t*>(uc + NBPC);        // [6][NBPF]
  constexpr int JF = (NBPF + kXferThreads - 1) / kXferThreads, JC = (NBPC + kXferThreads - 1) / kXferThreads;
  const int t = threadIdx.x;
  if (t < 8) sw[t] = wt.w[t];
  for (int e = t; e < 6 * NBPF / 8; e += kXferThreads)
    reinterpret_cast<uint4*>(ent)[e] = __ldg(reinterpret_cast<const uint4*>(tb.ent) + e);
  pdl_enter();
  for (int64_t b = blockIdx.x; b < n_blocks; b += gridDim.x) {
    __syncthreads();  // the tables are in; the previous block is done with uc
    const int up = __ldg(upper + b);
    // all of a thread's codes, then all of its values, are loaded together
    int32_t cc[JC], cf[JF];
#pragma unroll
    for (int q = 0; q < JC; ++q) {
      const int n = t + kXferThreads * q;
      cc[q] = n < NBPC ? __ldg(ccodes + b * NBPC + n) : -1;
    }
#pragma unroll
    for (int q = 0; q < JF; ++q) {
      const int n = t + kXferThreads * q;
      cf[q] = n < NBPF ? __ldg(fcodes + b * NBPF + n) : -1;
      if (n < NBPF && (__ldg(tb.hi + n) & up)) cf[q] = -1;
    }
    T vc[JC], vf[JF];
#pragma unroll
    for (int q = 0; q < JC; ++q) vc[q] = cc[q] >= 0 ? xc[cc[q] & 0x3FFFFFFF] : T(0);
#pragma unroll
    for (int q = 0; q < JF; ++q) vf[q] = cf[q] >= 0 ? xf[cf[q] & 0x3FFFFFFF] : T(0);
#pragma unroll
    for (int q = 0; q < JC; ++q)
      if (t + kXferThreads * q < NBPC) uc[t + kXferThreads * q] = vc[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < JF; ++q) {
      if (cf[q] < 0) continue;
      const int n = t + kXferThreads * q;
      double acc = 0.0;
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        const uint32_t v = ent[e * NBPF + n];
        if ((v >> 12) == 7) break;
        acc += sw[v >> 12] * double(uc[v & 0xFFF]);
      }
      xf[cf[q] & 0x3FFFFFFF] = vf[q] + T(acc);
    }
  }
}

// xc += P^T r, r = xf (MINUS: xf - tf, the residual formed on the way)
template <typename T, int NBPF, int NBPC, bool MINUS>
__global__ void __launch_bounds__(kXferThreads)
    block_restrict_add(int64_t n_blocks, const __grid_constant__ BlockTransferTables tb,
                       const __grid_constant__ BlockWeights wt, const uint8_t* __restrict__ upper,
                       const int32_t* __restrict__ fcodes, const int32_t* __restrict__ ccodes,
                       const T* xf, const T* tf, T* xc) {
  extern __shared__ __align__(16) unsigned char smem_x[];
  double* sw = reinterpret_cast<double*>(smem_x);          // [8]
  T* rf = reinterpret_cast<T*>(smem_x + 64);               // [NBPF]
  uint16_t* list = reinterpret_cast<uint16_t*>(rf + NBPF); // [n_list]
  constexpr int JF = (NBPF + kXferThreads - 1) / kXferThreads;
  const int t = threadIdx.x;
  if (t < 8) sw[t] = wt.w[t];
  for (int e = t; e < tb.n_list; e += kXferThreads) list[e] = __ldg(tb.list + e);
  pdl_enter();
  for (int64_t b = blockIdx.x; b < n_blocks; b += gridDim.x) {
    __syncthreads();  // the tables are in; the previous block is done with rf
    const int up = __ldg(upper + b);
    // all of a thread's codes, then all of its values, are loaded together
    int32_t cf[JF];
#pragma unroll
    for (int q = 0; q < JF; ++q) {
      const int n = t + kXferThreads * q;
      cf[q] = n < NBPF ? __ldg(fcodes + b * NBPF + n) : -1;
      if (n < NBPF && (__ldg(tb.hi + n) & up)) cf[q] = -1;
    }
    T v[JF], w[JF];
#pragma unroll
    for (int q = 0; q < JF; ++q) {
      v[q] = cf[q] >= 0 ? xf[cf[q] & 0x3FFFFFFF] : T(0);
      w[q] = MINUS && cf[q] >= 0 ? tf[cf[q] & 0x3FFFFFFF] : T(0);
    }
#pragma unroll
    for (int q = 0; q < JF; ++q)
      if (t + kXferThreads * q < NBPF) rf[t + kXferThreads * q] = v[q] - w[q];
    __syncthreads();
    for (int k = t; k < NBPC; k += kXferThreads) {
      const int n = __ldg(tb.order + k);
      const int32_t c = __ldg(ccodes + b * NBPC + n);
      if (c < 0) continue;
      double acc = 0.0;
      const int e1 = __ldg(tb.start + n + 1);
      for (int e = __ldg(tb.start + n); e < e1; ++e) {
        const uint32_t v = list[e];
        acc += sw[v >> 12] * double(rf[v & 0xFFF]);
      }
      T* d = xc + (c & 0x3FFFFFFF);
      if (c & 0x40000000) *d += T(acc);
      else if (acc != 0.0) atomicAdd(d, T(acc));
    }
  }
}

}  // namespace sfem
