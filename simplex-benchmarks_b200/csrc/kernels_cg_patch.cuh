// CG stiffness product by patches of consecutive cells, any mesh (sm_100a).
//
// A thread per cell that adds its K results atomically (cg_cell_kernel) sends K
// atomics a cell to L2 (P2: 10, of which each DoF of a tet mesh gets 7.5) and
// gathers as many values.  Here a CTA owns BS consecutive cells:
//   0. the distinct DoFs of the patch are gathered once into shared memory
//      (cp.async), while the lists of their contributions land next to them;
//   1. a thread per cell and component applies the cell operator; its results go to
//      shared memory by (local DoF, cell), where a warp writes without conflicts;
//   2. a lane per distinct DoF adds its contributions in a fixed order.  DoFs are
//      sorted by how many they have and dealt to warps 32 at a time, so the lanes of
//      a warp take the same number of steps.  DoFs no other patch has are stored, the
//      others added atomically.
// No mesh structure is used, only that consecutive cells are near one another.
// B200, unstructured, 44 x 40 x 36 hexes' cells, us per vmult with the fill of dst, thread per
// cell -> patches: P1 FP64 12.7 -> 8.4, FP32 12.8 -> 7.0; P2 FP64 22.7 -> 16.3, FP32 21.6 ->
// 11.9; P3 FP64 48.5 -> 46, FP32 46.9 -> 33; three components P2 FP64 63.7 -> 49.7, FP32 61.2
// -> 32.9.  P3 FP64 on 37 x 41 x 35 hexes 41 -> 35.  By the profiler (P2 FP64): the
// latency of the first loads (7 of 15 cycles an instruction at 12 to 14 warps per SM), L1
// 62 % (a third of the wavefronts are bank conflicts of the gather and the sums);
// atomics down from 10 to 3.1 a cell.
#pragma once
#include <cstdint>

#include "kernels_cg.cuh"
#include "kernels_dg_fused.cuh"

namespace sfem {

// Tables of all patches.  Slot 0 of a patch holds zero (constrained DoFs); distinct
// DoF s sits in slot 1 + s.
struct PatchTables {
  const uint32_t* slots;     // [patches][K / 2][BS]: slots of local DoFs 2 i, 2 i + 1
  const int32_t* ids;        // [patches][max_ids] distinct DoFs: DoF | no other patch has it << 30
  const int32_t* n_ids;      // [patches]
  const uint32_t* entries;   // per patch: first row of every 32 DoFs and the end, then rows of 32 pairs of entries
  const int32_t* ent_begin;  // [patches + 1] in units of 4 words
  int32_t max_ids, max_ent;
};
constexpr int32_t kPatchOwn = 0x40000000;

template <int P, int NC, int BS, typename T>
struct PatchShape {
  static constexpr int K = gen::Ops<P>::K;
  static constexpr int RS = K * BS + 1;  // results of a component, then a zero
  static constexpr int THREADS = BS * NC;
  static __host__ __device__ size_t bytes(int max_ids, int max_ent) {
    return size_t(max_ent) * 16 + (size_t(NC) * (max_ids + 1) + size_t(NC) * RS) * sizeof(T);
  }
};

template <int P, int NC, int BS, typename T, int MINB>
__global__ void __launch_bounds__(BS* NC, MINB)
    cg_patch_kernel(int64_t n_cells, const PatchTables tb, const T* __restrict__ geo, const T* __restrict__ src,
                    T* __restrict__ dst, int64_t n_constrained, const int32_t* __restrict__ constrained) {
  using S = PatchShape<P, NC, BS, T>;
  constexpr int K = S::K, THREADS = S::THREADS, PRE = 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t p = blockIdx.x;
  const int t = threadIdx.x, cell = t % BS, comp = t / BS;
  const int64_t c = p * BS + cell;
  uint32_t* se = reinterpret_cast<uint32_t*>(smem_raw);
  const int ms = tb.max_ids + 1;
  T* su = reinterpret_cast<T*>(smem_raw + size_t(tb.max_ent) * 16);  // [NC][ms]
  T* sy = su + NC * ms;                                              // [NC][RS]
  // the operator's own tables before the wait for src and dst
  const int32_t U = __ldg(tb.n_ids + p);
  const int32_t* ids = tb.ids + p * tb.max_ids;
  const int32_t e0 = __ldg(tb.ent_begin + p), ne = __ldg(tb.ent_begin + p + 1) - e0;
  uint32_t sl[K / 2];
  T G[6];
#pragma unroll
  for (int i = 0; i < K / 2; ++i) sl[i] = __ldg(tb.slots + (p * (K / 2) + i) * BS + cell);
  if (c < n_cells) {
#pragma unroll
    for (int k = 0; k < 6; ++k) G[k] = __ldg(geo + k * n_cells + c);
  }
  int32_t id[PRE];
#pragma unroll
  for (int r = 0; r < PRE; ++r) {
    const int e = t + r * THREADS;
    id[r] = e < tb.max_ids * NC ? __ldg(ids + e / NC) & ~kPatchOwn : 0;
  }
  for (int e = t; e < ne; e += THREADS) cp_async_bytes<16>(se + 4 * e, tb.entries + 4 * (int64_t(e0) + e));
  if (t < NC) {
    su[t * ms] = T(0);
    sy[t * S::RS + S::RS - 1] = T(0);
  }
  pdl_enter();
#pragma unroll
  for (int r = 0; r < PRE; ++r) {
    const int e = t + r * THREADS;
    if (e < U * NC) cp_async_bytes<sizeof(T)>(su + (e % NC) * ms + 1 + e / NC, src + int64_t(NC) * id[r] + e % NC);
  }
#pragma unroll 4
  for (int e = t + PRE * THREADS; e < U * NC; e += THREADS)
    cp_async_bytes<sizeof(T)>(su + (e % NC) * ms + 1 + e / NC,
                              src + int64_t(NC) * (__ldg(ids + e / NC) & ~kPatchOwn) + e % NC);
  cp_async_commit();
  for (int64_t k = p * THREADS + t; k < n_constrained; k += int64_t(gridDim.x) * THREADS) {
    const int32_t i = constrained[k];
    dst[i] = src[i];
  }
  cp_async_wait_all();
  __syncthreads();
  if (c < n_cells) {
    T u[K], y[K];
    const T* mine = su + comp * ms;
#pragma unroll
    for (int i = 0; i < K / 2; ++i) {
      u[2 * i] = mine[sl[i] & 0xFFFFu];
      u[2 * i + 1] = mine[sl[i] >> 16];
    }
    cg_local_apply<P>(G, u, y);
#pragma unroll
    for (int i = 0; i < K; ++i) sy[comp * S::RS + i * BS + cell] = y[i];
  }
  __syncthreads();
  const int lane = t % 32, chunks = (U + 31) / 32;
  for (int q = t / 32; q < chunks * NC; q += THREADS / 32) {
    const int ch = q / NC, k = q % NC, s = 32 * ch + lane;
    const int32_t g = s < U ? __ldg(ids + s) : 0;
    const T* row = sy + k * S::RS;
    const int r1 = int(se[ch + 1]);
    T sum = T(0);
#pragma unroll 2
    for (int r = int(se[ch]); r < r1; ++r) {
      const uint32_t e = se[32 * r + lane];
      sum += row[e & 0xFFFFu];
      sum += row[e >> 16];
    }
    if (s < U) {
      T* out = dst + int64_t(NC) * (g & ~kPatchOwn) + k;
      if (g & kPatchOwn) *out = sum;
      else atomicAdd(out, sum);
    }
  }
}

// Cells per CTA and resident CTAs that the registers are capped for.  44 x 40 x 36, us, by
// 64 / 128 / 256 cells: P1 FP64 9.5 / 8.5 / 9.2, P2 FP64 17.6 / 16.4 / 17.5, FP32 13.3 / 12.3 / 12.9;
// P3 FP64 by 32 / 64 / 128: 49.0 / 46.0 / 46.7; P2, three components, by 32 / 64 / 128: FP64 49.8 /
// 49.5 / 51.4, FP32 34.8 / 33.0 / 33.1.
template <int P, int NC>
__host__ __device__ constexpr int cg_patch_cells() {
  return NC == 3 ? 64 : 128;
}
template <int P, int NC, typename T>
__host__ __device__ constexpr int cg_patch_min_ctas() {
  constexpr int warps = cg_patch_cells<P, NC>() * NC / 32;
  return (P == 3 ? (sizeof(T) == 8 ? 12 : 20) : P == 2 ? (sizeof(T) == 8 ? 20 : 32) : 32) / warps;
}

}  // namespace sfem
