// Host tables of cg_block_kernel: a Kuhn box cut into 4 x 4 x 4-hex blocks.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

#include "../../include/simplex_fem.h"
#include "common.hpp"
#include "mesh.hpp"
#include "ref_tables.h"

namespace sfem {

struct CGBlockTables {
  int64_t n_blocks = 0;         // 0: the mesh is no Kuhn box (or too large for the codes)
  std::vector<int32_t> codes;   // [n_blocks][NBP]
  std::vector<uint8_t> upper;   // [n_blocks]: bit d set if the box goes on in direction d
  std::vector<int32_t> cell;    // [n_blocks][6][64]: cell of tet q of hex t, -1 where the box ends
};

// tet number of a cell of hex (i, j, k) from its ascending vertices' path along
// the hex edges (0..5 in the order of build_kuhn_mesh), -1 if it is no such path
inline int kuhn_tet(const Mesh& m, int64_t c, const int (&h)[3]) {
  static const int perms[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
  int at[3] = {h[0], h[1], h[2]}, axis[3];
  for (int v = 0; v < 4; ++v) {
    const auto L = m.vertex_lattice(m.cell_vertices[4 * c + v]);
    if (v > 0) {
      int a = -1;
      for (int d = 0; d < 3; ++d)
        if (L[d] == at[d] + 1 && a < 0) a = d;
      if (a < 0) return -1;
      axis[v - 1] = a;
      ++at[a];
    }
    for (int d = 0; d < 3; ++d)
      if (L[d] != at[d]) return -1;
  }
  for (int q = 0; q < 6; ++q)
    if (perms[q][0] == axis[0] && perms[q][1] == axis[1] && perms[q][2] == axis[2]) return q;
  return -1;
}

// lattice offsets of the nodes of the six tets of a hex
struct KuhnOffsets {
  int off[6][20][3] = {};
  explicit KuhnOffsets(int p) {
    static const int perms[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
    const int K = (p + 1) * (p + 2) * (p + 3) / 6;
    for (int q = 0; q < 6; ++q)
      for (int i = 0; i < K; ++i) {
        const int* a = p == 1 ? ref::Tables<1>::LATTICE[i] : p == 2 ? ref::Tables<2>::LATTICE[i] : ref::Tables<3>::LATTICE[i];
        int rest = a[1] + a[2] + a[3];
        for (int s = 0; s < 3; ++s) {
          off[q][i][perms[q][s]] = rest;
          rest -= a[s + 1];
        }
      }
  }
};

// Lattice node x + N1 (y + N1 z) of every slot: first-touch order of a full
// block's cells (hexes in Morton order), which is nearly the DoFs' order in
// memory.  Within windows of 128 slots the nodes are dealt to the groups of
// `span` lanes that share a shared-memory wavefront so that their banks
// (position mod nbank) differ where they can.
template <class At>
std::vector<int32_t> cg_block_slots(int p, int nbank, int span, At&& at) {
  const KuhnOffsets ko(p);
  const int K = (p + 1) * (p + 2) * (p + 3) / 6, N1 = 4 * p + 1, NB = N1 * N1 * N1;
  std::vector<int32_t> order;
  std::vector<char> seen(NB, 0);
  for (int h = 0; h < 64; ++h) {
    const int hx = (h & 1) | ((h >> 2) & 2), hy = ((h >> 1) & 1) | ((h >> 3) & 2), hz = ((h >> 2) & 1) | ((h >> 4) & 2);
    for (int q = 0; q < 6; ++q)
      for (int i = 0; i < K; ++i) {
        const int l = p * hx + ko.off[q][i][0] + N1 * (p * hy + ko.off[q][i][1] + N1 * (p * hz + ko.off[q][i][2]));
        if (!seen[l]) {
          seen[l] = 1;
          order.push_back(l);
        }
      }
  }
  SFEM_REQUIRE(int(order.size()) == NB, FEM_ERR_INTERNAL, "block tables: lattice");
  std::vector<int32_t> out;
  for (int w0 = 0; w0 < NB; w0 += 128) {
    const int len = std::min(128, NB - w0), groups = (len + span - 1) / span;
    std::vector<std::vector<int32_t>> g(groups);
    std::vector<std::vector<char>> used(groups, std::vector<char>(nbank, 0));
    std::vector<int32_t> rest;
    for (int e = w0; e < w0 + len; ++e) {
      const int l = order[e], bank = at(l % N1, (l / N1) % N1, l / (N1 * N1)) % nbank;
      int k = 0;
      while (k < groups && (used[k][bank] || int(g[k].size()) >= std::min(span, len - k * span))) ++k;
      if (k == groups) {
        rest.push_back(l);
        continue;
      }
      used[k][bank] = 1;
      g[k].push_back(l);
    }
    size_t r = 0;
    for (int k = 0; k < groups; ++k) {
      while (int(g[k].size()) < std::min(span, len - k * span)) g[k].push_back(rest[r++]);
      out.insert(out.end(), g[k].begin(), g[k].end());
    }
  }
  return out;
}

// cell_dofs [n_cells][K] of a continuous P_p numbering, constrained [n_dofs],
// lattice: cg_block_slots
inline CGBlockTables build_cg_block_tables(const Mesh& mesh, int p, const std::vector<int32_t>& cell_dofs,
                                           const std::vector<uint8_t>& constrained,
                                           const std::vector<int32_t>& lattice) {
  CGBlockTables T;
  const int* n = mesh.desc.n;
  const int64_t n_dofs = int64_t(constrained.size()), n_cells = mesh.n_cells;
  if (n_cells == 0 || n[0] < 1 || n[1] < 1 || n[2] < 1 || n_dofs >= (int64_t(1) << 30)) return T;
  if (mesh.n_vertices != int64_t(n[0] + 1) * (n[1] + 1) * (n[2] + 1)) return T;
  const int K = (p + 1) * (p + 2) * (p + 3) / 6, N1 = 4 * p + 1, NB = N1 * N1 * N1, NBP = (NB + 63) / 64 * 64;
  const KuhnOffsets ko(p);
  const auto& off = ko.off;
  std::vector<int32_t> slot(NB, -1);
  for (int e = 0; e < NB; ++e) slot[lattice[e]] = e;
  // cells of every block, blocks in the order of their first cell
  const int nb[3] = {(n[0] + 3) / 4, (n[1] + 3) / 4, (n[2] + 3) / 4};
  std::vector<int32_t> id(size_t(nb[0]) * nb[1] * nb[2], -1);
  int64_t blocks = 0;
  const int64_t n_hex = int64_t(n[0]) * n[1] * n[2];
  std::vector<int32_t> where(n_cells);  // 384 block + 64 q + t does not fit 31 bits for the largest boxes: kept apart
  std::vector<int16_t> place(n_cells);
  for (int64_t c = 0; c < n_cells; ++c) {
    const int64_t lin = mesh.cell_hex[c];
    if (lin < 0 || lin >= n_hex) return CGBlockTables{};
    const int h[3] = {int(lin % n[0]), int((lin / n[0]) % n[1]), int(lin / (int64_t(n[0]) * n[1]))};
    const int q = kuhn_tet(mesh, c, h);
    if (q < 0) return CGBlockTables{};
    int32_t& b = id[h[0] / 4 + int64_t(nb[0]) * (h[1] / 4 + int64_t(nb[1]) * (h[2] / 4))];
    if (b < 0) {
      b = int32_t(blocks++);
      uint8_t up = 0;
      for (int d = 0; d < 3; ++d) up |= uint8_t((h[d] / 4 + 1 < nb[d]) << d);
      T.upper.push_back(up);
    }
    where[c] = b;
    place[c] = int16_t(64 * q + (h[0] & 3) + 4 * (h[1] & 3) + 16 * (h[2] & 3));
  }
  T.cell.assign(size_t(384) * blocks, -1);
  for (int64_t c = 0; c < n_cells; ++c) {
    int32_t& e = T.cell[384 * size_t(where[c]) + place[c]];
    if (e >= 0) return CGBlockTables{};  // a tet listed twice
    e = int32_t(c);
  }
  std::vector<int32_t> count(n_dofs, 0);
  for (int32_t g : cell_dofs) ++count[g];
  T.codes.assign(size_t(NBP) * blocks, -1);
  bool ok = true;
#pragma omp parallel
  {
    std::vector<int32_t> dof(NB), local(NB);
#pragma omp for schedule(static)
    for (int64_t b = 0; b < blocks; ++b) {
      std::fill(dof.begin(), dof.end(), -1);
      std::fill(local.begin(), local.end(), 0);
      for (int q = 0; q < 6; ++q)
        for (int t = 0; t < 64; ++t) {
          const int64_t c = T.cell[384 * b + 64 * q + t];
          if (c < 0) continue;
          const int x = p * (t & 3), y = p * ((t >> 2) & 3), z = p * (t >> 4);
          for (int i = 0; i < K; ++i) {
            const int s = slot[x + off[q][i][0] + N1 * (y + off[q][i][1] + N1 * (z + off[q][i][2]))];
            const int32_t g = cell_dofs[size_t(K) * c + i];
            if (dof[s] >= 0 && dof[s] != g) ok = false;
            dof[s] = g;
            ++local[s];
          }
        }
      for (int s = 0; s < NB; ++s)
        if (dof[s] >= 0 && !constrained[dof[s]])
          T.codes[size_t(NBP) * b + s] = dof[s] | (local[s] == count[dof[s]] ? 0x40000000 : 0);
    }
  }
  if (!ok) return CGBlockTables{};
  T.n_blocks = blocks;
  return T;
}

}  // namespace sfem
