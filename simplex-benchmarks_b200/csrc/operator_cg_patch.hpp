// Tables and launch of cg_patch_kernel, for any tet mesh.
#pragma once
#include <algorithm>
#include <atomic>
#include <vector>

#include "kernels_cg_patch.cuh"
#include "operator.hpp"
#include "operator_parts.hpp"

namespace sfem {

template <typename T, int NC>
struct CGPatches {
  DevBuf<uint32_t> slots, entries;
  DevBuf<int32_t> ids, n_ids, ent_begin;
  PatchTables tb{};
  int64_t n_patches = 0, n_cells = 0, n_distinct = 0;
  // slots, distinct DoFs and lists that a product reads
  size_t table_bytes() const { return 4 * (slots.n + entries.n + size_t(n_distinct)); }

  static int cells_of(int p) {
    return p == 1 ? cg_patch_cells<1, NC>() : p == 2 ? cg_patch_cells<2, NC>() : cg_patch_cells<3, NC>();
  }
  static size_t smem_of(int p, int max_ids, int max_ent) {
    return p == 1   ? PatchShape<1, NC, cg_patch_cells<1, NC>(), T>::bytes(max_ids, max_ent)
           : p == 2 ? PatchShape<2, NC, cg_patch_cells<2, NC>(), T>::bytes(max_ids, max_ent)
                    : PatchShape<3, NC, cg_patch_cells<3, NC>(), T>::bytes(max_ids, max_ent);
  }

  // Below, SMs idle or take one patch more than others (B200, scalar, us per vmult,
  // patches / thread per cell: 192 patches (16^3 hexes) P1 FP64 4.1 / 4.0, P2 FP64 4.9 / 5.1,
  // P3 FP64 7.5 / 7.9, FP32 6.9 / 7.3; 159 patches P3 FP32 7.1 / 7.0; 375 patches (20^3) P1
  // FP64 4.2 / 4.5, P2 FP64 5.2 / 6.3, P3 FP32 7.9 / 9.6).
  static int min_patches(int p) { return p == 1 ? 256 : 192; }

  // cell_dofs [n_cells][K] node DoFs, constrained [nodes].  Leaves n_patches = 0 on
  // small meshes, where the tables' index bits do not suffice, and, unless the gathers
  // pay by themselves, where cells that follow one another are not neighbours: Morton order leaves 0.16 (P1), 0.29
  // (P2) and 0.39 (P3) distinct DoFs per cell and local DoF, rows of a box 0.41 for P3,
  // random order nearly one (24^3 hexes, patches / thread per cell: P2 FP64 10.3 / 9.4 us,
  // P3 FP64 23.4 / 16.2, P2 FP32 9.8 / 9.4, but P1 FP32 6.8 / 7.4, P3 FP32 14.8 / 19.3, three
  // components P2 FP32 17.7 / 22).  P1 has to have half of its cells' DoFs free: constrained
  // ones cost a thread per cell no gather and no atomic (1000 x 3 x 3 hexes, 44 % free: FP64
  // 4.4 / 4.1, three components 5.9 / 5.5; 400 x 400 x 1, none: 11.1 / 10.4; 200 x 100 x 2,
  // 50 %: 6.2 / 7.1; 1000 x 5 x 5, 64 %: 4.8 / 5.5).
  void build(int p, int K, int64_t nc, const std::vector<int32_t>& cell_dofs, const std::vector<uint8_t>& constrained) {
    if (nc == 0 || constrained.size() >= size_t(kPatchOwn)) return;
    const int BS = cells_of(p);
    const int64_t np = (nc + BS - 1) / BS;
    if (np < min_patches(p)) return;
    std::vector<int32_t> count(constrained.size(), 0);
    int64_t free = 0;
    for (int32_t g : cell_dofs) {
      ++count[g];
      free += !constrained[g];
    }
    if (p == 1 && double(free) < 0.47 * double(cell_dofs.size())) return;
    std::vector<uint32_t> sl(size_t(np) * (K / 2) * BS, 0);
    std::vector<std::vector<int32_t>> id(np);
    std::vector<std::vector<uint32_t>> en(np);
#pragma omp parallel
    {
      std::vector<uint64_t> key;
      struct Dof {
        int32_t g, first, n;
      };
      std::vector<Dof> dof;
#pragma omp for schedule(dynamic, 16)
      for (int64_t b = 0; b < np; ++b) {
        const int64_t c0 = b * BS, c1 = std::min(nc, c0 + BS);
        key.clear();
        dof.clear();
        for (int64_t c = c0; c < c1; ++c)
          for (int i = 0; i < K; ++i) {
            const int32_t g = cell_dofs[size_t(K) * c + i];
            if (!constrained[g]) key.push_back(uint64_t(g) << 32 | uint64_t(i * BS + (c - c0)));
          }
        std::sort(key.begin(), key.end());
        for (size_t e = 0; e < key.size(); ++e) {
          const int32_t g = int32_t(key[e] >> 32);
          if (dof.empty() || dof.back().g != g) dof.push_back({g, int32_t(e), 0});
          ++dof.back().n;
        }
        std::stable_sort(dof.begin(), dof.end(), [](const Dof& x, const Dof& y) { return x.n > y.n; });
        const int U = int(dof.size()), chunks = (U + 31) / 32;
        std::vector<uint32_t>& out = en[b];
        const int head = (chunks + 1 + 31) / 32;  // rows of 32 that the starts take
        out.assign(size_t(32) * head, 0);
        id[b].resize(U);
        for (int ch = 0; ch < chunks; ++ch) {
          const int rows = (dof[32 * ch].n + 1) / 2, r0 = int(out.size() / 32);
          out[ch] = uint32_t(r0);
          out.resize(out.size() + size_t(32) * rows, uint32_t(K * BS) * 0x10001u);  // the zero, twice
          for (int s = 32 * ch; s < std::min(U, 32 * ch + 32); ++s) {
            const Dof& d = dof[s];
            id[b][s] = d.g | (d.n == count[d.g] ? kPatchOwn : 0);
            for (int r = 0; r < d.n; ++r) {
              const uint32_t e = uint32_t(key[d.first + r]);
              uint32_t& pair = out[size_t(32) * (r0 + r / 2) + s % 32];
              pair = r % 2 ? (pair & 0xFFFFu) | e << 16 : (pair & 0xFFFF0000u) | e;
              const int i = int(e) / BS, cell = int(e) % BS;
              sl[(size_t(b) * (K / 2) + i / 2) * BS + cell] |= uint32_t(1 + s) << (16 * (i % 2));
            }
          }
        }
        out[chunks] = uint32_t(out.size() / 32);
      }
    }
    std::vector<int32_t> ni(np), eb(np + 1, 0);
    int64_t ne = 0, total = 0;
    for (int64_t b = 0; b < np; ++b) {
      tb.max_ids = std::max(tb.max_ids, int32_t(id[b].size()));
      tb.max_ent = std::max(tb.max_ent, int32_t(en[b].size() / 4));
      ni[b] = int32_t(id[b].size());
      total += ni[b];
      ne += int64_t(en[b].size() / 4);
      if (ne > INT32_MAX) return;
      eb[b + 1] = int32_t(ne);
    }
    if ((sizeof(T) == 8 || (NC == 1 && p == 2)) && 2 * total > int64_t(K) * nc) return;
    if (smem_of(p, tb.max_ids, tb.max_ent) > 200 * 1024) return;
    std::vector<int32_t> ai(size_t(np) * tb.max_ids, 0);
    std::vector<uint32_t> ae(4 * size_t(ne));
#pragma omp parallel for schedule(static)
    for (int64_t b = 0; b < np; ++b) {
      std::copy(id[b].begin(), id[b].end(), ai.begin() + b * tb.max_ids);
      std::copy(en[b].begin(), en[b].end(), ae.begin() + 4 * size_t(eb[b]));
    }
    slots.upload(sl);
    ids.upload(ai);
    n_ids.upload(ni);
    entries.upload(ae);
    ent_begin.upload(eb);
    tb.slots = slots.p;
    tb.ids = ids.p;
    tb.n_ids = n_ids.p;
    tb.entries = entries.p;
    tb.ent_begin = ent_begin.p;
    n_cells = nc;
    n_distinct = total;
    n_patches = np;
  }

  template <int P>
  void run(const T* geo, const T* x, T* d, int64_t n_constrained, const int32_t* constrained, cudaStream_t s) {
    constexpr int BS = cg_patch_cells<P, NC>();
    auto kern = cg_patch_kernel<P, NC, BS, T, cg_patch_min_ctas<P, NC, T>()>;
    static std::atomic<uint64_t> conf{0};
    int dev = 0;
    SFEM_CUDA(cudaGetDevice(&dev));
    once_per_device(conf, dev, [&] {
      SFEM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    });
    launch_pdl(kern, unsigned(n_patches), BS * NC, PatchShape<P, NC, BS, T>::bytes(tb.max_ids, tb.max_ent), s, n_cells,
               tb, geo, x, d, n_constrained, constrained);
  }
  void launch(int p, const T* geo, const T* x, T* d, int64_t n_constrained, const int32_t* constrained,
              cudaStream_t s) {
    switch (p) {
      case 1: run<1>(geo, x, d, n_constrained, constrained, s); break;
      case 2: run<2>(geo, x, d, n_constrained, constrained, s); break;
      case 3: run<3>(geo, x, d, n_constrained, constrained, s); break;
    }
    SFEM_CUDA(cudaGetLastError());
  }
};

}  // namespace sfem
