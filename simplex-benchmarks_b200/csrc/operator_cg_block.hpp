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
  BlockView view;  // also without the kernel: the multigrid's transfers go by blocks
  DevBuf<int16_t> pos;
  DevBuf<T> geo;
  int64_t n_blocks = 0, n_cells = 0;
  int grid = 0, resident = 0;  // resident: CTAs that the device holds at once

  // Whether the block form is the fastest one here.  A block costs the same however
  // many of its 64 hexes are there (boxes thinner than four hexes, sides that four
  // does not divide, a partition's cut), and a wave of blocks takes the time of one
  // block; patches (cg_patch_kernel), cells and, for P1, hexes cost by the hex.  B200,
  // us per vmult, block form / the fastest other one, hexes (per block):
  //   P1, from 10,000 hexes (9000 (36) FP64 4.5 / 4.1; 10,600 (49) 4.4 / 4.4) and 34
  //     (FP64) or 30 (FP32) per block: 160,000 (32) FP64 18.1 / 12.2, FP32 8.8 / 8.7;
  //     56,700 (36) FP64 6.4 / 7.1; 160,000 (16) FP64 30.9 / 9.8, FP32 16.7 / 7.6.
  //   P2 FP64, from 23,000: 21,952 (64) 8.2 / 7.3, 24,389 (48) 8.3 / 9.2; FP32 from
  //     31,000: 27,000 (53) 7.3 / 6.9, 32,400 (48) 7.6 / 8.4; both from 42 per block,
  //     38 where there are many: 50,000 (40) FP64 14.3 / 13.1, FP32 12.0 / 10.0;
  //     38,400 (48) 10.4 / 10.8, 8.2 / 8.8; 150,000 (39) 37.6 / 39.0, 23.7 / 25.9;
  //     160,000 (32) 47.3 / 38.2, 29.0 / 26.1.
  //   P3 FP32 by waves w, about 3.5 + 12 w us against 0.5 us per 1000 hexes: 27,000
  //     (one wave) 15.4 / 16.5, 35,937 (two) 26.5 / 18.1, 46,656 (two) 28.1 / 23.4,
  //     53,095 (two) 26.7 / 25.5, 68,921 (three) 37.2 / 34.4, 110,592 (three) 38.9 / 43.9.
  //   Three components, P1 from 10,000 and 24: 9000 (36) FP64 6.9 / 5.6, 25,000 (25) 8.5
  //     / 9.7.  P2 FP64 from 42 per block and 18,000, or whole blocks: 17,576 (51) 15.5 /
  //     14.2, 13,824 (64) 12.6 / 13.1, 20,800 (52) 15.6 / 16.8, 50,000 (40) 39.4 / 35.4.
  //     P2 FP32 from 36 and 16,000: 15,625 (46) 11.6 / 10.8, 17,576 (51) 11.6 / 11.7,
  //     40,000 (32) 22.0 / 20.5, 56,700 (36) 26.9 / 28.7.  P3 FP32 (no kernel): 46,656
  //     (64) 79 / 70, 110,592 (64) 168 / 160, thin boxes 2 / 1.
  bool pays(int p) const {
    if (!n_blocks) return false;
    const int64_t hexes = n_cells / 6;
    const bool f64 = sizeof(T) == 8;
    const double per = double(n_cells) / (6.0 * double(n_blocks));
    if (NC == 3)
      return p == 1 ? hexes >= 10000 && per >= 24
             : f64  ? per >= 60 || (per >= 42 && hexes >= 18000)
                    : per >= 36 && hexes >= 16000;
    if (p == 1) return hexes >= 10000 && per >= (f64 ? 34 : 30);
    if (p == 2) return hexes >= (f64 ? 23000 : 31000) && per >= (n_blocks >= 3000 ? 38 : 42);
    return hexes >= 30000 * ((n_blocks + resident - 1) / resident) - 6000;
  }

  std::vector<int32_t> cell;  // of every block's hexes' tets, until the metric by blocks is made

  // everything but the metric by blocks
  void build(const Mesh& mesh, int p, const std::vector<int32_t>& cell_dofs, const std::vector<uint8_t>& constrained) {
    const std::vector<int32_t> lattice = p == 1 ? slots<1>() : p == 2 ? slots<2>() : slots<3>();
    CGBlockTables tb = build_cg_block_tables(mesh, p, cell_dofs, constrained, lattice);
    if (!tb.n_blocks) return;
    codes.upload(tb.codes);
    upper.upload(tb.upper);
    view.n_blocks = tb.n_blocks;
    view.codes = codes.p;
    view.upper = upper.p;
    view.lattice = lattice;
    if (!has_kernel(p)) return;
    n_blocks = tb.n_blocks;
    n_cells = mesh.n_cells;
    cell = std::move(tb.cell);
    switch (p) {
      case 1: setup<1>(lattice); break;
      case 2: setup<2>(lattice); break;
      case 3:
        if constexpr (has_kernel(3)) setup<3>(lattice);
        break;
    }
  }
  // the metric by blocks, as large as the operator's own: made where the form runs
  void make_metric(const DevBuf<T>& d_geo) {
    if (!n_blocks || geo.n) return;
    const std::vector<T> soa = d_geo.download();  // [6][n_cells]
    std::vector<T> g(size_t(36) * 64 * n_blocks);
#pragma omp parallel for schedule(static)
    for (int64_t b = 0; b < n_blocks; ++b)
      for (int q = 0; q < 6; ++q)
        for (int t = 0; t < 64; ++t) {
          const int64_t c = cell[384 * b + 64 * q + t];
          for (int k = 0; k < 6; ++k)
            g[(36 * size_t(b) + 6 * q + k) * 64 + t] = c >= 0 ? soa[size_t(k) * n_cells + c] : T(0);
        }
    geo.upload(g);
    SFEM_CUDA(cudaStreamSynchronize(nullptr));  // other streams do not wait for the copy
    cell = {};
  }
  // codes and metric that a product reads
  size_t table_bytes() const { return codes.n * sizeof(int32_t) + size_t(36) * 64 * n_blocks * sizeof(T); }
  // P3 FP64 (two resident CTAs of 64 threads): never the faster one (64^3 177 us, cubes
  // 143 us; three components 48^3 392, a thread per cell 226 us), nor P3 FP32 with three
  // components
  static constexpr bool has_kernel(int p) { return p <= 2 || (sizeof(T) == 4 && NC == 1); }

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
    resident = sms * occ;
    grid = int(std::min<int64_t>(n_blocks, resident));
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
        if constexpr (has_kernel(3)) launch<3>(x, d, n_constrained, constrained, s);
        break;
    }
    SFEM_CUDA(cudaGetLastError());
  }
};

}  // namespace sfem
