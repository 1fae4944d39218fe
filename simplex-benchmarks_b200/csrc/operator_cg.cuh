// Continuous Galerkin operators: set-up (geometry, index tables) and kernel
// dispatch.  A template on the number type, instantiated by operator_cg_f64.cu
// and operator_cg_f32.cu.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <unordered_map>

#include "kernels_cg.cuh"
#include "kernels_cg_tc.cuh"
#include "kernels_dg.cuh"
#include "op_shapes.hpp"
#include "operator.hpp"
#include "operator_cg_block.hpp"
#include "operator_cg_patch.hpp"
#include "operator_parts.hpp"

namespace sfem {

namespace {

// ------------------------------------------------------------------ CG ----
template <typename T>
class CGOperator final : public Operator {
 public:
  DevBuf<int32_t> d_dofs;        // [K][n_cells], -1 = constrained
  DevBuf<T> d_geo;               // [6][n_cells]
  DevBuf<int32_t> d_constrained; // constrained DoF list
  // macro-element (hex) tables of cg_hex_kernel, made by make_hex_tables; hex_H = 0
  // when the mesh is not 6 consecutive Kuhn tets per hex with one common DoF pattern
  DevBuf<int32_t> d_hdofs;       // [H][n_hex]
  DevBuf<T> d_hgeo;              // [36][n_hex]: metric of tet q at rows 6 q .. 6 q + 5
  HexMap hex_map{};
  int64_t n_hex = 0;
  int hex_H = 0;

  static int hex_dofs(int p) { return p == 1 ? 8 : p == 2 ? 27 : 64; }

  // TF32 tensor-core tables (variant 4, FP32 operators): B = [S_0; ..; S_5]
  DevBuf<float> d_btc;
  DevBuf<int> d_status;
  int tc_grid = 0;

  // (S_c)_ij of the cell operator y = sum_c G_c S_c u over the metric
  // components c = (00,11,22,01,02,12): S_aa = D_a^T MQ D_a,
  // S_ab = D_a^T MQ D_b + D_b^T MQ D_a
  template <int P>
  static double stiffness_S(int c, int i, int j) {
    using Tb = ref::Tables<P>;
    constexpr int KQ = Tb::KQ;
    static const int ca[6] = {0, 1, 2, 0, 0, 1}, cb[6] = {0, 1, 2, 1, 2, 2};
    auto E = [&](int a, int b) {
      double s = 0;
      for (int m = 0; m < KQ; ++m)
        for (int q = 0; q < KQ; ++q) s += Tb::D[a][m][i] * Tb::MQ[m][q] * Tb::D[b][q][j];
      return s;
    };
    return ca[c] == cb[c] ? E(ca[c], cb[c]) : E(ca[c], cb[c]) + E(cb[c], ca[c]);
  }
  // round to TF32 (10 mantissa bits, nearest, ties away)
  static float tf32_round(double v) {
    float f = float(v);
    uint32_t bits;
    std::memcpy(&bits, &f, 4);
    bits = (bits + 0x1000u) & 0xFFFFE000u;
    std::memcpy(&f, &bits, 4);
    return f;
  }

  template <int P>
  void build_tc_tables() {
    using Sh = CGTcShape<P>;
    std::vector<float> B(size_t(Sh::NPAD) * Sh::KPAD, 0.0f);
    for (int c = 0; c < 6; ++c)
      for (int i = 0; i < Sh::K; ++i)
        for (int j = 0; j < Sh::K; ++j) B[size_t(c * Sh::K + i) * Sh::KPAD + j] = tf32_round(stiffness_S<P>(c, i, j));
    d_btc.upload(B);
    int dev = 0, sms = 0, occ = 0;
    SFEM_CUDA(cudaGetDevice(&dev));
    SFEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SFEM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, cg_cell_tc_kernel<P>, 128, Sh::SMEM_BYTES));
    occ = std::min(occ, 512 / Sh::TMEM_COLS);  // tensor-memory columns per SM
    SFEM_REQUIRE(occ > 0, FEM_ERR_CUDA, "CG tensor-core kernel does not fit on an SM");
    tc_grid = int(std::min<int64_t>((n_cells + 127) / 128, int64_t(sms) * occ));
  }

  int status(bool clear) override {
    if (!d_status.p) return 0;
    int v = 0;
    SFEM_CUDA(cudaMemcpy(&v, d_status.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (clear && v) SFEM_CUDA(cudaMemset(d_status.p, 0, sizeof(int)));
    return v;
  }

  // 4 x 4 x 4-hex blocks of cg_block_kernel; empty on meshes that are no Kuhn boxes
  CGBlocks<T, 1> blocks;
  // patches of cells of cg_patch_kernel, where a thread per cell is the default
  CGPatches<T, 1> patches;

  // cube-block tables of cg_cube_kernel (blocks of 64 hexes = 384 tets)
  DevBuf<int16_t> d_tmapv, d_cslot8[3];
  DevBuf<uint32_t> d_ritem[3];
  DevBuf<int32_t> d_bdof;
  int64_t n_blocks = 0;
  int cube_NB = 0;
  static int cube_nb(int p) { return p == 1 ? 125 : p == 2 ? 729 : 2197; }
  static int cube_kp(int k) { return (k % 2) ? k : k + 1; }

  void build_cube_tables(const CGDofs& dofs) {
    if (n_cells == 0 || n_cells % 384 != 0) return;
    const int NB = cube_nb(cfg.degree), KP = cube_kp(K);
    const int64_t nbk = n_cells / 384;
    // cube-local numbering by first occurrence over (tet, local DoF)
    auto local = [&](int64_t b, std::vector<int16_t>& tm, std::vector<int32_t>& order,
                     std::unordered_map<int32_t, int>& at) -> bool {
      order.clear();
      at.clear();
      tm.resize(size_t(384) * K);
      for (int t = 0; t < 384; ++t)
        for (int i = 0; i < K; ++i) {
          const int32_t g = dofs.cell_dofs[size_t(K) * (384 * b + t) + i];
          auto it = at.find(g);
          int j;
          if (it == at.end()) {
            j = int(order.size());
            if (j >= NB) return false;
            at.emplace(g, j);
            order.push_back(g);
          } else {
            j = it->second;
          }
          tm[t * K + i] = int16_t(j);
        }
      return int(order.size()) == NB;
    };
    std::vector<int16_t> tm0;
    std::vector<int32_t> ord0;
    std::unordered_map<int32_t, int> at0;
    if (!local(0, tm0, ord0, at0)) return;
    // contribution lists and their sizes (identical in every block)
    std::vector<std::vector<int16_t>> contrib(NB);
    for (int t = 0; t < 384; ++t)
      for (int i = 0; i < K; ++i) contrib[tm0[t * K + i]].push_back(int16_t(t * KP + i));
    // reduce slots: slot n = 384 r + 32 w + l is gathered and reduced by lane
    // l of warp w in round r.  DoFs sorted by contribution groups of 8
    // (most first; first-occurrence order inside a class, which keeps the
    // global addresses of a warp's gathers and stores close) form chunks of
    // 32 that fill one warp-round each, so the lanes of a warp loop over the
    // same number of groups; the chunks are dealt longest-first to the
    // least-loaded warp, which balances the warps up to the block barrier.
    std::vector<int> jorder(NB), slot_of(NB), dof_at(NB);
    for (int j = 0; j < NB; ++j) jorder[j] = j;
    std::stable_sort(jorder.begin(), jorder.end(), [&](int a, int b2) {
      return (contrib[a].size() + 7) / 8 > (contrib[b2].size() + 7) / 8;
    });
    {
      constexpr int NW = 12;
      const int NJr = (NB + 383) / 384, nch = (NB + 31) / 32;
      std::vector<int> cap(NW, 0), used(NW, 0), load(NW, 0), base(nch, -1);
      for (int r = 0; r < NJr; ++r)
        for (int w = 0; w < NW; ++w) {
          const int len = std::max(0, std::min(32, NB - (384 * r + 32 * w)));
          if (len == 32) ++cap[w];
          else if (len > 0) base[nch - 1] = 384 * r + 32 * w;  // the one partial chunk
        }
      auto cost = [&](int c) {
        int mx = 0;
        for (int e = 32 * c; e < std::min(NB, 32 * c + 32); ++e) mx = std::max(mx, int(contrib[jorder[e]].size()));
        return mx + 2 * ((mx + 7) / 8) + 4;
      };
      std::vector<int> corder;
      for (int c = 0; c < nch; ++c)
        if (base[c] < 0) corder.push_back(c);
      std::stable_sort(corder.begin(), corder.end(), [&](int a, int b2) { return cost(a) > cost(b2); });
      for (int c : corder) {
        int w = -1;
        for (int v = 0; v < NW; ++v)
          if (used[v] < cap[v] && (w < 0 || load[v] < load[w])) w = v;
        SFEM_REQUIRE(w >= 0, FEM_ERR_INTERNAL, "cube tables: no warp-round left for a chunk");
        base[c] = 384 * used[w] + 32 * w;
        ++used[w];
        load[w] += cost(c);
      }
      for (int e = 0; e < NB; ++e) {
        slot_of[jorder[e]] = base[e / 32] + e % 32;
        dof_at[base[e / 32] + e % 32] = jorder[e];
      }
    }
    std::vector<int32_t> count(m, 0);
    for (size_t i = 0; i < dofs.cell_dofs.size(); ++i) ++count[dofs.cell_dofs[i]];
    std::vector<int32_t> bd(size_t(NB) * nbk);
    bool ok = true;
#pragma omp parallel
    {
      std::vector<int16_t> tm;
      std::vector<int32_t> ord;
      std::unordered_map<int32_t, int> at;
      at.reserve(4 * NB);
#pragma omp for schedule(dynamic, 16)
      for (int64_t b = 0; b < nbk; ++b) {
        if (!ok) continue;
        if (!local(b, tm, ord, at) || tm != tm0) {
          ok = false;
          continue;
        }
        for (int n = 0; n < NB; ++n) {
          const int j = dof_at[n];
          const int32_t g = ord[j];
          const bool interior = count[g] == int(contrib[j].size());
          bd[size_t(b) * NB + n] = dofs.constrained[g] ? -1 : (g | (interior ? 0x40000000 : 0));
        }
      }
    }
    if (!ok || m >= (int64_t(1) << 30)) return;
    // packed tables, laid out so that a warp reads 16 consecutive bytes per
    // lane:
    //   tmapv  [KV/8][384] x 8 int16: slot of tet t's local DoF i (KV = K
    //          rounded up to 8, padding entries 0);
    //   cslot8 per warp-round, [groups][32 lanes] x 8 int16: the row slot
    //          (t' * KP + i) each lane reads at each step;
    //   ritem  [NB]: steps of the lane | (first cslot8 entry << 8).
    // Three reduce schedules (kernel variants 5, 6, 7):
    //   0  each lane reads its contributions in (tet, local DoF) order;
    //   1  bank-scheduled, the same steps for every lane of a warp-round;
    //   2  bank-scheduled, each lane stops after its last contribution.
    // Bank-scheduled steps come from an edge colouring of the bipartite
    // multigraph lanes x shared-memory banks (one edge per contribution): a
    // bipartite multigraph of maximum degree D has a proper D-edge-colouring
    // (Konig), found here by alternating-path recolouring.  Colour = step, so
    // no two lanes of one step hit the same bank and every step is one
    // shared-memory wavefront (per half-warp for 8-byte values).  A lane with
    // nothing to add at a step reads one of the zero slots 384 * KP + z (one
    // per bank), in a bank that no other lane of the step uses.
    const int KV = (K + 7) / 8 * 8;
    std::vector<int16_t> tmv(size_t(384) * KV, 0);
    for (int t = 0; t < 384; ++t)
      for (int i = 0; i < K; ++i) tmv[(size_t(i / 8) * 384 + t) * 8 + i % 8] = int16_t(slot_of[tm0[t * K + i]]);
    const int nbank = sizeof(T) == 8 ? 16 : 32;  // 8-byte values: 16 bank pairs per half-warp
    const int span = sizeof(T) == 8 ? 16 : 32;   // lanes that share one wavefront
    SFEM_REQUIRE(384 * KP + 32 < 32768, FEM_ERR_INTERNAL, "cube tables exceed their index bits");
    for (int mode = 0; mode < 3; ++mode) {
      std::vector<int16_t> c8;
      std::vector<uint32_t> items(NB);
      for (int n0 = 0; n0 < NB; n0 += 32) {
        const int len = std::min(32, NB - n0);
        std::vector<std::vector<int>> step_slot(32);  // per lane: slot at each step, -1 = none
        for (int h0 = 0; h0 < len; h0 += span) {
          const int h1 = std::min(len, h0 + span);
          if (mode == 0) {
            for (int l = h0; l < h1; ++l)
              for (int16_t v : contrib[dof_at[n0 + l]]) step_slot[l].push_back(v);
            continue;
          }
          std::vector<std::pair<int, int>> edges;  // (lane in span, slot)
          std::vector<int> degl(span, 0), degb(nbank, 0);
          for (int l = h0; l < h1; ++l)
            for (int16_t v : contrib[dof_at[n0 + l]]) {
              edges.emplace_back(l - h0, v);
              ++degl[l - h0];
              ++degb[v % nbank];
            }
          const int D = std::max(*std::max_element(degl.begin(), degl.end()),
                                 *std::max_element(degb.begin(), degb.end()));
          std::vector<int> Lc(size_t(span) * D, -1), Bc(size_t(nbank) * D, -1), col(edges.size(), -1);
          auto lc = [&](int u, int c) -> int& { return Lc[size_t(u) * D + c]; };
          auto bc = [&](int v, int c) -> int& { return Bc[size_t(v) * D + c]; };
          for (size_t e = 0; e < edges.size(); ++e) {
            const int u = edges[e].first, v = edges[e].second % nbank;
            int a = 0, c2 = 0;
            while (lc(u, a) >= 0) ++a;
            while (bc(v, c2) >= 0) ++c2;
            if (a != c2 && bc(v, a) >= 0) {
              // swap colours a and c2 along the alternating path that leaves bank v by colour a
              std::vector<int> path;
              bool at_bank = true;
              int node = v, c = a;
              for (;;) {
                const int ed = at_bank ? bc(node, c) : lc(node, c);
                if (ed < 0) break;
                path.push_back(ed);
                node = at_bank ? edges[ed].first : edges[ed].second % nbank;
                at_bank = !at_bank;
                c = c == a ? c2 : a;
              }
              for (int ed : path) {
                lc(edges[ed].first, col[ed]) = -1;
                bc(edges[ed].second % nbank, col[ed]) = -1;
              }
              for (int ed : path) {
                col[ed] = col[ed] == a ? c2 : a;
                lc(edges[ed].first, col[ed]) = ed;
                bc(edges[ed].second % nbank, col[ed]) = ed;
              }
            }
            SFEM_REQUIRE(lc(u, a) < 0 && bc(v, a) < 0, FEM_ERR_INTERNAL, "cube tables: edge colouring failed");
            col[e] = a;
            lc(u, a) = int(e);
            bc(v, a) = int(e);
          }
          for (size_t e = 0; e < edges.size(); ++e) {
            std::vector<int>& st = step_slot[h0 + edges[e].first];
            if (int(st.size()) <= col[e]) st.resize(col[e] + 1, -1);
            st[col[e]] = edges[e].second;
          }
        }
        int S = 0;
        for (int l = 0; l < len; ++l) S = std::max(S, int(step_slot[l].size()));
        SFEM_REQUIRE(S > 0 && S < 256, FEM_ERR_INTERNAL, "cube tables: step count out of range");
        std::vector<int> steps(len);
        for (int l = 0; l < len; ++l) {
          steps[l] = mode == 1 ? S : int(step_slot[l].size());
          step_slot[l].resize(S, -1);
        }
        // gaps: a zero slot in a bank that no lane of the span reads at that step
        for (int h0 = 0; h0 < len; h0 += span) {
          const int h1 = std::min(len, h0 + span);
          for (int st = 0; st < S; ++st) {
            std::vector<char> busy(nbank, 0);
            for (int l = h0; l < h1; ++l)
              if (step_slot[l][st] >= 0) busy[step_slot[l][st] % nbank] = 1;
            const int f = int(std::find(busy.begin(), busy.end(), 0) - busy.begin());
            for (int l = h0; l < h1; ++l)
              if (step_slot[l][st] < 0) step_slot[l][st] = 384 * KP + ((f % nbank - 384 * KP) % nbank + nbank) % nbank;
          }
        }
        const size_t e0 = c8.size() / 8;
        c8.resize(c8.size() + size_t((S + 7) / 8) * 32 * 8, int16_t(384 * KP));
        for (int l = 0; l < len; ++l) {
          for (int e = 0; e < S; ++e) c8[((e0 + size_t(e / 8) * 32) + l) * 8 + e % 8] = int16_t(step_slot[l][e]);
          items[n0 + l] = uint32_t(steps[l]) | (uint32_t(e0 + l) << 8);
        }
      }
      SFEM_REQUIRE(c8.size() / 8 < (size_t(1) << 24), FEM_ERR_INTERNAL, "cube tables exceed their index bits");
      d_ritem[mode].upload(items);
      d_cslot8[mode].upload(c8);
    }
    d_tmapv.upload(tmv);
    d_bdof.upload(bd);
    n_blocks = nbk;
    cube_NB = NB;
  }

  void launch_tc_cell(const T* x, T* d, cudaStream_t s) {
    const float* xf = reinterpret_cast<const float*>(x);
    float* df = reinterpret_cast<float*>(d);
    switch (cfg.degree) {
      case 1: cg_cell_tc_kernel<1><<<tc_grid, 128, CGTcShape<1>::SMEM_BYTES, s>>>(n_cells, d_dofs.p, reinterpret_cast<const float*>(d_geo.p), d_btc.p, xf, df, d_constrained.n, d_constrained.p, d_status.p); break;
      case 2: cg_cell_tc_kernel<2><<<tc_grid, 128, CGTcShape<2>::SMEM_BYTES, s>>>(n_cells, d_dofs.p, reinterpret_cast<const float*>(d_geo.p), d_btc.p, xf, df, d_constrained.n, d_constrained.p, d_status.p); break;
      case 3: cg_cell_tc_kernel<3><<<tc_grid, 128, CGTcShape<3>::SMEM_BYTES, s>>>(n_cells, d_dofs.p, reinterpret_cast<const float*>(d_geo.p), d_btc.p, xf, df, d_constrained.n, d_constrained.p, d_status.p); break;
    }
    SFEM_CUDA(cudaGetLastError());
  }

  int cube_grid = 0;
  template <int P, int NB, int KP>
  static size_t cube_smem() {
    return ((cube_metric_smem<P, T>() ? 6 * 384 : 0) + 2 * size_t(NB) + 384 * size_t(KP) + (sizeof(T) == 8 ? 16 : 32)) *
           sizeof(T);
  }
  template <int P, int NB, int KP>
  void setup_cube() {
    auto kern = cg_cube_pipe_kernel<P, T, NB, KP>;
    SFEM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(cube_smem<P, NB, KP>())));
    int dev = 0, sms = 0, occ = 0;
    SFEM_CUDA(cudaGetDevice(&dev));
    SFEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SFEM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 384, cube_smem<P, NB, KP>()));
    SFEM_REQUIRE(occ > 0, FEM_ERR_CUDA, "CG cube kernel does not fit on an SM");
    cube_grid = int(std::min<int64_t>(n_blocks, int64_t(sms) * occ));
  }
  template <int P, int NB, int KP>
  void launch_cube(const T* x, T* d, int sched, cudaStream_t s) {
    launch_pdl(cg_cube_pipe_kernel<P, T, NB, KP>, unsigned(cube_grid), 384, cube_smem<P, NB, KP>(), s, n_blocks,
               d_tmapv.p, d_bdof.p, d_ritem[sched].p, d_cslot8[sched].p, d_geo.p, x, d, int64_t(d_constrained.n),
               d_constrained.p);
  }

  // TF32 tensor-core cube kernel (variant 8, FP32 operators with cube tables):
  // B rows p NP + n = (S_c)_i. for c = p CPP + n / K, i = n % K
  DevBuf<float> d_bcube;
  int cube_tc_grid = 0;
  size_t cube_tc_smem = 0;
  template <int P, int NB, int KP>
  void setup_cube_tc() {
    using Sh = CubeTcShape<P>;
    std::vector<float> B(size_t(Sh::NBROWS) * Sh::KPAD, 0.0f);
    for (int p = 0; p < Sh::PASSES; ++p)
      for (int n = 0; n < Sh::CPP * Sh::K; ++n)
        for (int j = 0; j < Sh::K; ++j)
          B[size_t(p * Sh::NP + n) * Sh::KPAD + j] = tf32_round(stiffness_S<P>(p * Sh::CPP + n / Sh::K, n % Sh::K, j));
    d_bcube.upload(B);
    auto kern = cg_cube_tc_kernel<P, NB, KP>;
    int dev = 0, sms = 0, occ = 0;
    SFEM_CUDA(cudaGetDevice(&dev));
    SFEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // more CTAs per SM than the tensor memory holds would wait in tcgen05.alloc
    // for another CTA to finish: pad the shared memory until they cannot fit
    size_t smem = Sh::smem_bytes(NB, KP);
    for (;;) {
      SFEM_REQUIRE(smem <= 227 * 1024, FEM_ERR_CUDA, "CG tensor-core cube kernel: no shared-memory size fits");
      SFEM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
      SFEM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 384, smem));
      if (occ <= Sh::MAX_CTAS) break;
      smem += 4096;
    }
    SFEM_REQUIRE(occ > 0, FEM_ERR_CUDA, "CG tensor-core cube kernel does not fit on an SM");
    cube_tc_smem = smem;
    cube_tc_grid = int(std::min<int64_t>(n_blocks, int64_t(sms) * occ));
  }
  template <int P, int NB, int KP>
  void launch_cube_tc(const T* x, T* d, int sched, cudaStream_t s) {
    cg_cube_tc_kernel<P, NB, KP><<<unsigned(cube_tc_grid), 384, cube_tc_smem, s>>>(
        n_blocks, d_tmapv.p, d_bdof.p, d_ritem[sched].p, d_cslot8[sched].p, reinterpret_cast<const float*>(d_geo.p),
        d_bcube.p, reinterpret_cast<const float*>(x), reinterpret_cast<float*>(d), d_constrained.n, d_constrained.p,
        d_status.p);
  }

  // whether the mesh is 6 consecutive Kuhn tets per hex with one common DoF pattern
  void find_hex_pattern(const Mesh& mesh, const CGDofs& dofs) {
    if (n_cells == 0 || n_cells % 6 != 0 || int64_t(mesh.cell_hex.size()) != n_cells) return;
    const int64_t nh = n_cells / 6;
    const int H = hex_dofs(cfg.degree);
    // hex-local numbering by first occurrence over (tet, local DoF)
    auto local_map = [&](int64_t h, int8_t (&mm)[6][20], std::vector<int32_t>& order) -> bool {
      order.clear();
      for (int q = 0; q < 6; ++q) {
        if (mesh.cell_hex[6 * h + q] != mesh.cell_hex[6 * h]) return false;
        for (int i = 0; i < K; ++i) {
          const int32_t g = dofs.cell_dofs[size_t(K) * (6 * h + q) + i];
          int k = 0;
          while (k < int(order.size()) && order[k] != g) ++k;
          if (k == int(order.size())) {
            if (k >= H) return false;
            order.push_back(g);
          }
          mm[q][i] = int8_t(k);
        }
      }
      return int(order.size()) == H;
    };
    HexMap m0{};
    std::vector<int32_t> ord0;
    if (!local_map(0, m0.m, ord0)) return;
    bool ok = true;
#pragma omp parallel
    {
      std::vector<int32_t> ord;
      int8_t mm[6][20];
#pragma omp for schedule(static)
      for (int64_t h = 0; h < nh; ++h) {
        if (!ok) continue;
        bool same = local_map(h, mm, ord);
        for (int q = 0; q < 6 && same; ++q)
          for (int i = 0; i < K; ++i) same = same && mm[q][i] == m0.m[q][i];
        if (!same) ok = false;
      }
    }
    if (!ok) return;
    hex_map = m0;
    n_hex = nh;
    hex_H = H;
  }

  // the hex form's DoF and metric tables, as large as the operator's own
  void make_hex_tables() {
    if (!hex_H || d_hdofs.n) return;
    int first[64];  // tet and local DoF of every hex-local DoF
    for (int q = 5; q >= 0; --q)
      for (int i = K - 1; i >= 0; --i) first[hex_map.m[q][i]] = q * K + i;
    const std::vector<T> geo = d_geo.download();
    std::vector<int32_t> hd(size_t(hex_H) * n_hex);
    std::vector<T> hg(36 * size_t(n_hex));
#pragma omp parallel for schedule(static)
    for (int64_t h = 0; h < n_hex; ++h) {
      for (int k = 0; k < hex_H; ++k) {
        const int32_t g = cell_dofs[size_t(K) * 6 * h + first[k]];
        hd[size_t(k) * n_hex + h] = constrained[g] ? -1 : g;
      }
      for (int q = 0; q < 6; ++q)
        for (int k = 0; k < 6; ++k) hg[size_t(6 * q + k) * n_hex + h] = geo[size_t(k) * n_cells + 6 * h + q];
    }
    d_hgeo.upload(hg);
    d_hdofs.upload(hd);
    SFEM_CUDA(cudaStreamSynchronize(nullptr));  // other streams do not wait for the copies
  }

  // the tables that only variant v's form reads
  void make_tables(int v) {
    if (v == 0) v = default_form;
    if (v == 3 && use_blocks()) blocks.make_metric(d_geo);
    else if (v == 2 || ((v == 3 || (v >= 5 && v <= 7)) && !cube_NB)) make_hex_tables();
  }
  std::mutex tables_mutex;
  void set_variant(int v) override {
    {
      std::lock_guard<std::mutex> lock(tables_mutex);
      RelaxedCapture relaxed;
      make_tables(v);
    }
    cfg.kernel_variant = v;
  }

  CGOperator(const Mesh& mesh, const OpConfig& c) : CGOperator(mesh, build_cg_dofs(mesh, c.degree), nullptr, c) {}

  // Operator on the cells of `mesh` with a given numbering: dofs.constrained
  // masks the gather and scatter, `identity` (default: dofs.constrained)
  // lists the rows that get dst = src.  A partition's local operator passes
  // the global constraints of its owned and ghost DoFs and only the owned
  // constrained DoFs as identity rows.
  CGOperator(const Mesh& mesh, CGDofs dofs, const std::vector<uint8_t>* identity, const OpConfig& c) {
    cfg = c;
    if (cfg.weak_bc) {
      // weak (Nitsche) Dirichlet: no DoF is constrained, boundary faces carry
      // the penalty terms instead
      std::fill(dofs.constrained.begin(), dofs.constrained.end(), uint8_t(0));
      identity = nullptr;
    }
    K = dofs.K;
    n_cells = mesh.n_cells;
    m = dofs.n_dofs;
    n_interior_faces = mesh.n_interior_faces;
    n_boundary_faces = mesh.n_boundary_faces;
    cell_dofs = dofs.cell_dofs;
    constrained = dofs.constrained;
    support = dofs.support;
    std::vector<int32_t> idx(size_t(K) * n_cells);
    for (int64_t cc = 0; cc < n_cells; ++cc)
      for (int i = 0; i < K; ++i) {
        const int32_t g = dofs.cell_dofs[K * cc + i];
        idx[size_t(i) * n_cells + cc] = dofs.constrained[g] ? -1 : g;
      }
    d_dofs.upload(idx);
    std::vector<T> geo(6 * size_t(n_cells));
    for (int64_t cc = 0; cc < n_cells; ++cc) {
      double G[6];
      metric(cell_geometry(mesh, cc), G);
      for (int k = 0; k < 6; ++k) geo[size_t(k) * n_cells + cc] = T(G[k]);
    }
    d_geo.upload(geo);
    std::vector<int32_t> cl;
    const std::vector<uint8_t>& id_rows = identity ? *identity : constrained;
    SFEM_REQUIRE(int64_t(id_rows.size()) == m, FEM_ERR_INTERNAL, "CG: identity mask size");
    for (int64_t i = 0; i < m; ++i)
      if (id_rows[i]) cl.push_back(int32_t(i));
    d_constrained.upload(cl);
    find_hex_pattern(mesh, dofs);
    build_cube_tables(dofs);
    blocks.build(mesh, cfg.degree, dofs.cell_dofs, dofs.constrained);
    default_form = default_variant();
    if (default_form == 1) patches.build(cfg.degree, K, n_cells, dofs.cell_dofs, dofs.constrained);
    if (cfg.weak_bc) build_weak_boundary(mesh);
    d_status.alloc(1);
    SFEM_CUDA(cudaMemset(d_status.p, 0, sizeof(int)));
    if (std::is_same<T, float>::value && n_cells > 0) {
      switch (cfg.degree) {
        case 1: build_tc_tables<1>(); break;
        case 2: build_tc_tables<2>(); break;
        case 3: build_tc_tables<3>(); break;
      }
    }
    if (cube_NB) {
      switch (cfg.degree) {
        case 1: setup_cube<1, 125, 5>(); break;
        case 2: setup_cube<2, 729, 11>(); break;
        case 3: setup_cube<3, 2197, 21>(); break;
      }
      if (std::is_same<T, float>::value) {
        switch (cfg.degree) {
          case 1: setup_cube_tc<1, 125, 5>(); break;
          case 2: setup_cube_tc<2, 729, 11>(); break;
          case 3: setup_cube_tc<3, 2197, 21>(); break;
        }
      }
    }
    if (hex_H) {
      switch (cfg.degree) {
        case 1: setup_hex<1, 8>(); break;
        case 2: setup_hex<2, 27>(); break;
        case 3: setup_hex<3, 64>(); break;
      }
    }
    make_tables(cfg.kernel_variant);
  }

  static constexpr int kHexBS = 64;
  template <int P, int H>
  static size_t hex_smem() { return 2 * size_t(kHexBS) * HexRow<H>::S * sizeof(T); }
  template <int P, int H>
  void setup_hex() {
    SFEM_CUDA(cudaFuncSetAttribute(cg_hex_kernel<P, T, H, kHexBS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(hex_smem<P, H>())));
  }
  template <int P, int H>
  void launch_hex(const T* x, T* d, cudaStream_t s) {
    const unsigned grid = blocks_for(std::max<int64_t>(n_hex, 1), kHexBS);
    cg_hex_kernel<P, T, H, kHexBS><<<grid, kHexBS, hex_smem<P, H>(), s>>>(
        n_hex, d_hdofs.p, hex_map, d_hgeo.p, x, d, d_constrained.n, d_constrained.p);
  }

  void vmult(void* dst, const void* src, cudaStream_t s) override {
    vmult_phase(dst, src, 1, s);
    vmult_phase(dst, src, 2, s);
  }
  bool needs_zero() const override { return true; }
  void vmult_zeroed(void* dst, const void* src, cudaStream_t s) override { vmult_phase(dst, src, 2, s); }

  void vmult_phase(void* dst, const void* src, int phase, cudaStream_t s) override {
    T* d = static_cast<T*>(dst);
    const T* x = static_cast<const T*>(src);
    if (phase == 1) {
      SFEM_CUDA(cudaMemsetAsync(d, 0, sizeof(T) * m, s));
      return;
    }
    apply_cells(x, d, s);
    if (cfg.weak_bc) apply_boundary(x, d, false, s);
  }

  // weak (Nitsche) boundary terms: boundary faces grouped by local face number
  DevBuf<int32_t> d_bcell[4];
  DevBuf<T> d_bsf[4];

  void build_weak_boundary(const Mesh& mesh) {
    const int p = cfg.degree;
    const double factor = double((p + 1) * (p + 3)) / 3.0;
    std::vector<int32_t> cells[4];
    std::vector<T> sf[4];
    for (int64_t cc = 0; cc < n_cells; ++cc) {
      const double vol = std::fabs(cell_geometry(mesh, cc).det) / 6.0;
      double area[4], surf = 0;
      for (int f = 0; f < 4; ++f) {
        double nrm[3];
        face_area_normal(mesh, cc, f, area[f], nrm);
        surf += area[f] * (mesh.nb[4 * cc + f] == -1 ? 1.0 : 0.5);
      }
      const double tau = surf / vol;  // surface / volume (DG/cells_batched/application_phc.cc:1284-1313)
      for (int f = 0; f < 4; ++f)
        if (mesh.nb[4 * cc + f] == -1) {
          cells[f].push_back(int32_t(cc));
          sf[f].push_back(T(factor * tau * area[f]));
        }
    }
    for (int f = 0; f < 4; ++f) {
      d_bcell[f].upload(cells[f]);
      d_bsf[f].upload(sf[f]);
    }
  }

  template <int P>
  void launch_boundary(const T* x, T* d, bool diag, cudaStream_t s) {
    auto go = [&](auto fc) {
      constexpr int F = decltype(fc)::value;
      const int64_t nb = int64_t(d_bcell[F].n);
      if (!nb) return;
      cg_weak_boundary_kernel<P, F, T><<<blocks_for(nb, 128), 128, 0, s>>>(nb, d_bcell[F].p, d_bsf[F].p, n_cells,
                                                                          d_dofs.p, d_geo.p, x, d, diag);
    };
    go(std::integral_constant<int, 0>{});
    go(std::integral_constant<int, 1>{});
    go(std::integral_constant<int, 2>{});
    go(std::integral_constant<int, 3>{});
  }

  void apply_boundary(const T* x, T* d, bool diag, cudaStream_t s) {
    switch (cfg.degree) {
      case 1: launch_boundary<1>(x, d, diag, s); break;
      case 2: launch_boundary<2>(x, d, diag, s); break;
      case 3: launch_boundary<3>(x, d, diag, s); break;
    }
    SFEM_CUDA(cudaGetLastError());
  }

  // Variant 3: block form (cg_block_kernel) or thread-per-tet cube kernel, where both
  // apply.  P1 and P2: always the block form.  P3 FP32: the block form where it pays or
  // there are no whole cubes (a wave of blocks takes 15 us: 36^3 28.1, cubes 23.6 us).
  bool use_blocks() const {
    return blocks.n_blocks && (cfg.degree <= 2 || !cube_NB || blocks.pays(cfg.degree));
  }
  // Variant 0: the block form where it pays; cubes for P3 (two per SM at least: 28^3
  // FP32 14.4, patches 14.9 us); P1 boxes with too little in a block go by hexes once
  // there are many (2 x 200 x 400: FP64 hexes 12.2, patches 14.8 us; 48^3 9.4 / 11.7, but
  // 37^3 7.1 / 7.5, 32^3 6.6 / 5.9); else 1, which is cg_patch_kernel if the mesh has
  // enough patches (CGPatches), or a thread per cell.  P3 FP64 without whole cubes: 37 x
  // 41 x 35 hexes 41.5 us by cells, per hex 49.5 us.
  int default_form = 1;  // default_variant(), once at set-up
  int default_variant() const {
    if (blocks.pays(cfg.degree)) return 3;
    if (cfg.degree == 3 && cube_NB && n_blocks >= 2 * 148) return 3;
    if (cfg.degree == 1 && hex_H && n_hex >= 50000) return 2;
    return 1;
  }

  void apply_cells(const T* x, T* d, cudaStream_t s) {
    int v = cfg.kernel_variant;
    if (v == 8) {
      // TF32 tensor cores per cube; per cell (variant 4) without whole cubes
      SFEM_REQUIRE(d_btc.p != nullptr, FEM_ERR_ARG, "CG kernel variant 8 (TF32 tensor cores) needs an FP32 operator");
      if (cube_NB && cube_tc_grid) {
        switch (cfg.degree) {
          case 1: launch_cube_tc<1, 125, 5>(x, d, 0, s); break;
          case 2: launch_cube_tc<2, 729, 11>(x, d, 0, s); break;
          case 3: launch_cube_tc<3, 2197, 21>(x, d, 0, s); break;
        }
        SFEM_CUDA(cudaGetLastError());
        return;
      }
      v = 4;
    }
    if (v == 4) {
      SFEM_REQUIRE(d_btc.p != nullptr, FEM_ERR_ARG, "CG kernel variant 4 (TF32 tensor cores) needs an FP32 operator");
      launch_tc_cell(x, d, s);
      return;
    }
    if (v == 0) v = default_form;
    // variant 3: the block form where it is the faster one, else the cube kernel;
    // cube reduce schedule: variants 5, 6, 7 pick one; variant 3 takes the one
    // measured fastest on B200 (FP64 P1 and P2: bank-scheduled with uniform steps;
    // FP32 and P3: contribution order)
    int sched = v >= 5 ? v - 5 : (sizeof(T) == 8 && cfg.degree <= 2 ? 1 : 0);
    if (v == 3 && use_blocks()) {
      blocks.launch(cfg.degree, x, d, d_constrained.n, d_constrained.p, s);
      return;
    }
    if (v >= 5) v = 3;
    if (v == 3 && cube_NB) {
      switch (cfg.degree) {
        case 1: launch_cube<1, 125, 5>(x, d, sched, s); break;
        case 2: launch_cube<2, 729, 11>(x, d, sched, s); break;
        case 3: launch_cube<3, 2197, 21>(x, d, sched, s); break;
      }
      SFEM_CUDA(cudaGetLastError());
      return;
    }
    // variant 2 (and 3 without whole cubes): one thread per hex; the cell
    // kernel on meshes without the common hex pattern
    if ((v == 2 || v == 3) && hex_H) {
      switch (cfg.degree) {
        case 1: launch_hex<1, 8>(x, d, s); break;
        case 2: launch_hex<2, 27>(x, d, s); break;
        case 3: launch_hex<3, 64>(x, d, s); break;
      }
      SFEM_CUDA(cudaGetLastError());
      return;
    }
    if (v == 1 && patches.n_patches) {
      patches.launch(cfg.degree, d_geo.p, x, d, d_constrained.n, d_constrained.p, s);
      return;
    }
    const int64_t n = std::max<int64_t>(n_cells, int64_t(d_constrained.n));
    const unsigned grid = blocks_for(n, 128);
    switch (cfg.degree) {
      case 1: launch_pdl(cg_cell_kernel<1, T>, grid, 128, 0, s, n_cells, d_dofs.p, d_geo.p, x, d, int64_t(d_constrained.n), d_constrained.p); break;
      case 2: launch_pdl(cg_cell_kernel<2, T>, grid, 128, 0, s, n_cells, d_dofs.p, d_geo.p, x, d, int64_t(d_constrained.n), d_constrained.p); break;
      case 3:
        // P3 in FP64: registers capped for 4 CTAs per SM (measured faster on B200)
        if (sizeof(T) == 8) launch_pdl(cg_cell_kernel<3, T, 4>, grid, 128, 0, s, n_cells, d_dofs.p, d_geo.p, x, d, int64_t(d_constrained.n), d_constrained.p);
        else launch_pdl(cg_cell_kernel<3, T>, grid, 128, 0, s, n_cells, d_dofs.p, d_geo.p, x, d, int64_t(d_constrained.n), d_constrained.p);
        break;
    }
    SFEM_CUDA(cudaGetLastError());
  }

  void diagonal(void* diag, cudaStream_t s) override {
    T* d = static_cast<T*>(diag);
    SFEM_CUDA(cudaMemsetAsync(d, 0, sizeof(T) * m, s));
    const int64_t n = std::max<int64_t>(n_cells, int64_t(d_constrained.n));
    const unsigned grid = blocks_for(n, 128);
    switch (cfg.degree) {
      case 1: cg_diagonal_kernel<1, T><<<grid, 128, 0, s>>>(n_cells, d_dofs.p, d_geo.p, d, d_constrained.n, d_constrained.p); break;
      case 2: cg_diagonal_kernel<2, T><<<grid, 128, 0, s>>>(n_cells, d_dofs.p, d_geo.p, d, d_constrained.n, d_constrained.p); break;
      case 3: cg_diagonal_kernel<3, T><<<grid, 128, 0, s>>>(n_cells, d_dofs.p, d_geo.p, d, d_constrained.n, d_constrained.p); break;
    }
    SFEM_CUDA(cudaGetLastError());
    if (cfg.weak_bc) apply_boundary(nullptr, d, true, s);
  }

  const int32_t* device_dof_table() const override { return d_dofs.p; }
  bool block_form() const override { return use_blocks() && blocks.n_blocks >= 148; }
  // default variant; 3 is the block form, cubes, hexes; 1 is the patch form
  std::string forms() const override {
    return std::to_string(default_form) + (use_blocks() ? "b" : "") + (cube_NB ? "c" : "") + (hex_H ? "h" : "") +
           (patches.n_patches ? "p" : "");
  }
  const BlockView* block_view() const override { return blocks.view.n_blocks ? &blocks.view : nullptr; }

  void element_matrices(void* out, cudaStream_t s) override {
    T* m = static_cast<T*>(out);
    const unsigned grid = blocks_for(std::max<int64_t>(n_cells, 1), 128);
    switch (cfg.degree) {
      case 1: cg_element_matrix_kernel<1, T><<<grid, 128, 0, s>>>(n_cells, d_geo.p, m); break;
      case 2: cg_element_matrix_kernel<2, T><<<grid, 128, 0, s>>>(n_cells, d_geo.p, m); break;
      case 3: cg_element_matrix_kernel<3, T><<<grid, 128, 0, s>>>(n_cells, d_geo.p, m); break;
    }
    SFEM_CUDA(cudaGetLastError());
  }

  void work(double& flops, double& bytes) const override {
    const int p = cfg.degree, kq = kq_of(p);
    const double per_cell = 2.0 * (2 * nnz_grad_rt(p) + 9 * kq + 3 * kq * kq);
    flops = per_cell * double(n_cells);
    bytes = 2.0 * sizeof(T) * double(m) + double(table_bytes());
  }
  // index and metric tables that the current form reads
  size_t table_bytes() const {
    const size_t metric = d_geo.n * sizeof(T);
    const int v = cfg.kernel_variant == 0 ? default_form : cfg.kernel_variant;
    if (v == 3 && use_blocks()) return blocks.table_bytes();
    if ((v == 3 || v >= 5) && cube_NB) return metric + d_bdof.n * sizeof(int32_t);
    if (v == 2 || v == 3 || (v >= 5 && v <= 7))
      if (hex_H) return metric + size_t(hex_H) * n_hex * sizeof(int32_t);
    if (v == 1 && patches.n_patches) return metric + patches.table_bytes();
    return metric + d_dofs.n * sizeof(int32_t);
  }
};

// ------------------------------------------------------- CG, 3 components --
// Vector Laplacian with the components of every node DoF interleaved
// (index 3 g + comp), as the reference's components-batched CG operator
// (CG/components_batched/application.cc:778-1611, FESystem of dim
// FE_SimplexP).  Homogeneous Dirichlet on every component of the boundary
// nodes.  cg_block_kernel on Kuhn boxes, else cg_patch_kernel or a thread per cell.
template <typename T>
class CGVectorOperator final : public Operator {
 public:
  static constexpr int NC = 3;
  DevBuf<int32_t> d_dofs;         // [K][n_cells] node DoFs, -1 = constrained
  DevBuf<T> d_geo;                // [6][n_cells]
  DevBuf<int32_t> d_constrained;  // constrained vector indices
  int64_t n_nodes = 0;
  std::vector<int32_t> node_dofs;  // [n_cells][K]
  CGBlocks<T, NC> blocks;          // 4 x 4 x 4-hex blocks (Kuhn boxes)
  CGPatches<T, NC> patches;        // patches of cells elsewhere
  bool blocks_pay = false;         // the block form is the default

  CGVectorOperator(const Mesh& mesh, const OpConfig& c) {
    cfg = c;
    const CGDofs dofs = build_cg_dofs(mesh, cfg.degree);
    K = dofs.K;
    n_cells = mesh.n_cells;
    n_nodes = dofs.n_dofs;
    m = NC * n_nodes;
    n_interior_faces = mesh.n_interior_faces;
    n_boundary_faces = mesh.n_boundary_faces;
    node_dofs = dofs.cell_dofs;
    cell_dofs.resize(size_t(NC) * K * n_cells);
    for (int64_t cc = 0; cc < n_cells; ++cc)
      for (int comp = 0; comp < NC; ++comp)
        for (int i = 0; i < K; ++i)
          cell_dofs[(cc * NC + comp) * K + i] = NC * dofs.cell_dofs[K * cc + i] + comp;
    constrained.assign(m, 0);
    std::vector<int32_t> cl;
    for (int64_t g = 0; g < n_nodes; ++g)
      if (dofs.constrained[g])
        for (int comp = 0; comp < NC; ++comp) {
          constrained[NC * g + comp] = 1;
          cl.push_back(int32_t(NC * g + comp));
        }
    support = dofs.support;
    std::vector<int32_t> idx(size_t(K) * n_cells);
    for (int64_t cc = 0; cc < n_cells; ++cc)
      for (int i = 0; i < K; ++i) {
        const int32_t g = dofs.cell_dofs[K * cc + i];
        idx[size_t(i) * n_cells + cc] = dofs.constrained[g] ? -1 : g;
      }
    d_dofs.upload(idx);
    std::vector<T> geo(6 * size_t(n_cells));
    for (int64_t cc = 0; cc < n_cells; ++cc) {
      double G[6];
      metric(cell_geometry(mesh, cc), G);
      for (int k = 0; k < 6; ++k) geo[size_t(k) * n_cells + cc] = T(G[k]);
    }
    d_geo.upload(geo);
    d_constrained.upload(cl);
    blocks.build(mesh, cfg.degree, dofs.cell_dofs, dofs.constrained);
    blocks_pay = blocks.pays(cfg.degree);
    make_tables(cfg.kernel_variant);
    // P3 FP64 keeps the thread per cell: 44 x 40 x 36 hexes 130 us, by patches 137 to 160
    if (!blocks_pay && (cfg.degree <= 2 || sizeof(T) == 4))
      patches.build(cfg.degree, K, n_cells, dofs.cell_dofs, dofs.constrained);
  }
  void make_tables(int v) {
    if (v == 3 || (v == 0 && blocks_pay)) blocks.make_metric(d_geo);
  }
  std::mutex tables_mutex;
  void set_variant(int v) override {
    {
      std::lock_guard<std::mutex> lock(tables_mutex);
      RelaxedCapture relaxed;
      make_tables(v);
    }
    cfg.kernel_variant = v;
  }
  bool block_form() const override { return blocks.n_blocks >= 148; }
  std::string forms() const override {
    return std::string(blocks_pay ? "3" : "1") + (blocks.n_blocks ? "b" : "") +
           (patches.n_patches ? "p" : "");
  }

  void vmult(void* dst, const void* src, cudaStream_t s) override {
    vmult_phase(dst, src, 1, s);
    vmult_phase(dst, src, 2, s);
  }

  void vmult_phase(void* dst, const void* src, int phase, cudaStream_t s) override {
    T* d = static_cast<T*>(dst);
    const T* x = static_cast<const T*>(src);
    if (phase == 1) {
      SFEM_CUDA(cudaMemsetAsync(d, 0, sizeof(T) * m, s));
      return;
    }
    const int v = cfg.kernel_variant;
    if (blocks.n_blocks && (v == 3 || (v == 0 && blocks_pay))) {
      blocks.launch(cfg.degree, x, d, d_constrained.n, d_constrained.p, s);
      return;
    }
    if (patches.n_patches) {
      patches.launch(cfg.degree, d_geo.p, x, d, d_constrained.n, d_constrained.p, s);
      return;
    }
    const unsigned grid = blocks_for(std::max<int64_t>(n_cells, int64_t(d_constrained.n)), 128);
    switch (cfg.degree) {
      case 1: launch_pdl(cg_cell_vec_kernel<1, T, NC>, grid, 128, 0, s, n_cells, d_dofs.p, d_geo.p, x, d, int64_t(d_constrained.n), d_constrained.p); break;
      case 2: launch_pdl(cg_cell_vec_kernel<2, T, NC>, grid, 128, 0, s, n_cells, d_dofs.p, d_geo.p, x, d, int64_t(d_constrained.n), d_constrained.p); break;
      case 3: launch_pdl(cg_cell_vec_kernel<3, T, NC>, grid, 128, 0, s, n_cells, d_dofs.p, d_geo.p, x, d, int64_t(d_constrained.n), d_constrained.p); break;
    }
    SFEM_CUDA(cudaGetLastError());
  }

  void diagonal(void* diag, cudaStream_t s) override {
    DevBuf<T> dn(n_nodes);
    SFEM_CUDA(cudaMemsetAsync(dn.p, 0, sizeof(T) * n_nodes, s));
    std::vector<int32_t> cn;
    for (int64_t g = 0; g < n_nodes; ++g)
      if (constrained[NC * g]) cn.push_back(int32_t(g));
    DevBuf<int32_t> d_cn;
    d_cn.upload(cn);
    const unsigned grid = blocks_for(std::max<int64_t>(n_cells, int64_t(cn.size())), 128);
    switch (cfg.degree) {
      case 1: cg_diagonal_kernel<1, T><<<grid, 128, 0, s>>>(n_cells, d_dofs.p, d_geo.p, dn.p, d_cn.n, d_cn.p); break;
      case 2: cg_diagonal_kernel<2, T><<<grid, 128, 0, s>>>(n_cells, d_dofs.p, d_geo.p, dn.p, d_cn.n, d_cn.p); break;
      case 3: cg_diagonal_kernel<3, T><<<grid, 128, 0, s>>>(n_cells, d_dofs.p, d_geo.p, dn.p, d_cn.n, d_cn.p); break;
    }
    expand_components<T, NC><<<blocks_for(std::max<int64_t>(n_nodes, 1), 256), 256, 0, s>>>(
        n_nodes, dn.p, static_cast<T*>(diag));
    SFEM_CUDA(cudaGetLastError());
    SFEM_CUDA(cudaStreamSynchronize(s));  // the temporaries are freed on return
  }

  void rhs(const RhsDesc& rd, void* dst, cudaStream_t s) override {
    throw Error(FEM_ERR_ARG, "rhs: not provided for the 3-component CG operator");
  }

  void work(double& flops, double& bytes) const override {
    const int p = cfg.degree, kq = kq_of(p);
    flops = NC * 2.0 * (2 * nnz_grad_rt(p) + 9 * kq + 3 * kq * kq) * double(n_cells);
    const int v = cfg.kernel_variant;
    const bool by_blocks = blocks.n_blocks && (v == 3 || (v == 0 && blocks_pay));
    const size_t tables = by_blocks ? blocks.table_bytes()
                                    : d_geo.n * sizeof(T) + (patches.n_patches ? patches.table_bytes()
                                                                               : d_dofs.n * sizeof(int32_t));
    bytes = 2.0 * sizeof(T) * double(m) + double(tables);
  }
};

}  // namespace

template <typename T>
std::unique_ptr<Operator> make_cg_operator(const Mesh& mesh, const OpConfig& cfg) {
  if (cfg.n_components == 3) return std::make_unique<CGVectorOperator<T>>(mesh, cfg);
  return std::make_unique<CGOperator<T>>(mesh, cfg);
}
template <typename T>
std::unique_ptr<Operator> make_cg_local_operator(const Mesh& mesh, const CGDofs& dofs,
                                                 const std::vector<uint8_t>* identity, const OpConfig& cfg) {
  return std::make_unique<CGOperator<T>>(mesh, dofs, identity, cfg);
}

}  // namespace sfem
