// Device tables and launch of cg_block_kernel, shared by the scalar and the
// three-component CG operators.
#pragma once
#include <algorithm>
#include <vector>

#include "cg_block_tables.hpp"
#include "kernels_cg_block.cuh"
#include "operator.hpp"

namespace sfem {

// Resident CTAs of 64 threads per SM that the registers are capped for (P2 FP64
// 168 registers, six CTAs; at 196 registers and five CTAs 128^3 takes 320 us
// instead of 285; P3 FP32 at 168 registers 97 instead of 89 us on 64^3).
template <int P, typename T>
constexpr int cg_block_min_ctas() {
  return P == 1 ? 8 : P == 2 ? (sizeof(T) == 8 ? 5 : 8) : 4;
}

template <typename T, int NC>
struct CGBlocks {
  DevBuf<int32_t> codes;
  DevBuf<uint8_t> upper;
  BlockView view;  // also without the kernel (P3 FP64): the multigrid's transfers go by blocks
  DevBuf<int16_t> pos;
  DevBuf<T> geo;
  int64_t n_blocks = 0;
  int grid = 0;

  // geo_soa: metric values [6][n_cells] in the operator's precision
  void build(const Mesh& mesh, int p, const std::vector<int32_t>& cell_dofs, const std::vector<uint8_t>& constrained,
             const std::vector<T>& geo_soa) {
    const std::vector<int32_t> lattice = p == 1 ? slots<1>() : p == 2 ? slots<2>() : slots<3>();
    const CGBlockTables tb = build_cg_block_tables(mesh, p, cell_dofs, constrained, lattice);
    if (!tb.n_blocks) return;
    codes.upload(tb.codes);
    upper.upload(tb.upper);
    view.n_blocks = tb.n_blocks;
    view.codes = codes.p;
    view.upper = upper.p;
    view.lattice = lattice;
    if (p == 3 && sizeof(T) == 8) return;  // the slower kernel there (see CGOperator::use_blocks)
    std::vector<T> g(size_t(36) * 64 * tb.n_blocks);
#pragma omp parallel for schedule(static)
    for (int64_t b = 0; b < tb.n_blocks; ++b)
      for (int q = 0; q < 6; ++q)
        for (int t = 0; t < 64; ++t) {
          const int64_t c = tb.cell[384 * b + 64 * q + t];
          for (int k = 0; k < 6; ++k)
            g[(36 * size_t(b) + 6 * q + k) * 64 + t] = c >= 0 ? geo_soa[size_t(k) * mesh.n_cells + c] : T(0);
        }
    geo.upload(g);
    n_blocks = tb.n_blocks;
    switch (p) {
      case 1: setup<1>(lattice); break;
      case 2: setup<2>(lattice); break;
      case 3:
        if constexpr (sizeof(T) == 4) setup<3>(lattice);
        break;
    }
  }

  template <int P>
  static constexpr auto kernel() {
    return cg_block_kernel<P, T, NC, cg_block_min_ctas<P, T>()>;
  }

  template <int P>
  static std::vector<int32_t> slots() {
    const int w = sizeof(T) == 8 ? 16 : 32;  // banks of the value size, lanes of a wavefront
    return cg_block_slots(P, w, w, [](int x, int y, int z) { return CGBlockShape<P, T>::at(x, y, z); });
  }

  template <int P>
  void setup(const std::vector<int32_t>& lattice) {
    using S = CGBlockShape<P, T>;
    std::vector<int16_t> p16(S::NBP, int16_t(S::LAT));  // padding entries write the spare slot
    for (int n = 0; n < S::NB; ++n) {
      const int l = lattice[n];
      p16[n] = int16_t(S::at(l % S::N1, (l / S::N1) % S::N1, l / (S::N1 * S::N1)));
    }
    pos.upload(p16);
    const size_t bytes = S::bytes(NC);
    int dev = 0, sms = 0, occ = 0;
    SFEM_CUDA(cudaGetDevice(&dev));
    SFEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SFEM_CUDA(cudaFuncSetAttribute(kernel<P>(), cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
    SFEM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel<P>(), 64, bytes));
    SFEM_REQUIRE(occ > 0, FEM_ERR_CUDA, "CG block kernel does not fit on an SM");
    grid = int(std::min<int64_t>(n_blocks, int64_t(sms) * occ));
  }

  template <int P>
  void launch(const T* x, T* d, int64_t n_constrained, const int32_t* constrained, cudaStream_t s) const {
    launch_pdl(kernel<P>(), unsigned(grid), 64, CGBlockShape<P, T>::bytes(NC), s, n_blocks, codes.p, pos.p, geo.p, x, d,
               n_constrained, constrained);
  }
  void launch(int p, const T* x, T* d, int64_t n_constrained, const int32_t* constrained, cudaStream_t s) const {
    switch (p) {
      case 1: launch<1>(x, d, n_constrained, constrained, s); break;
      case 2: launch<2>(x, d, n_constrained, constrained, s); break;
      case 3:
        if constexpr (sizeof(T) == 4) launch<3>(x, d, n_constrained, constrained, s);
        break;
    }
    SFEM_CUDA(cudaGetLastError());
  }
};

}  // namespace sfem
