// DG and Helmholtz operators: set-up (geometry, penalties, neighbours), kernel
// dispatch and the batched launch.  A template on the number type, instantiated
// by operator_dg_f64.cu and operator_dg_f32.cu.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>

#include "autotune.hpp"
#include "kernels_dg.cuh"
#include "kernels_dg2.cuh"
#include "kernels_dg3.cuh"
#include "kernels_dg_fused.cuh"
#include "kernels_dg_fused3.cuh"
#include "op_shapes.hpp"
#include "operator.hpp"
#include "operator_parts.hpp"

namespace sfem {

namespace {

// ------------------------------------------------------------------ DG ----
template <typename T>
class DGOperator final : public Operator {
 public:
  // for the two-launch forms and the diagonal (made by need_geometry)
  DevBuf<T> d_geo;      // [6 + 4 + (mass?1:0)][n_cells]
  DevBuf<int32_t> d_nb; // [4][n_cells]
  DevBuf<int8_t> d_nbf; // [4][n_cells]
  // single-launch forms (kernels_dg_fused.cuh, kernels_dg_fused3.cuh)
  DevBuf<unsigned char> d_fgeo;  // geometry by blocks of cells
  DevBuf<int32_t> d_ext_begin, d_ext;  // outer neighbours of every block
  int n_ext = 0;            // most of a block
  DevBuf<int32_t> d_face_begin;          // P3: outer faces of every block
  DevBuf<OuterFace<T>> d_outer;
  int n_outer = 0;
  DevBuf<T> d_Q;        // published face normal derivatives: [n_cells][4][NC][NFQ], or block-major
                        // (scalar problems, 1-thread-per-cell forms), for whole 128-cell blocks; made by
                        // need_traces
  DevBuf<int> d_status; // timeouts of the bounded waits in the bulk-copy trace pass
  bool has_mass = false;

  DGOperator(const Mesh& mesh, const OpConfig& c) {
    cfg = c;
    const int p = cfg.degree;
    K = k_of(p);
    n_cells = mesh.n_cells;
    m = int64_t(K) * cfg.n_components * n_cells;
    n_interior_faces = mesh.n_interior_faces;
    n_boundary_faces = mesh.n_boundary_faces;
    has_mass = cfg.kind == FEM_HELMHOLTZ;
    constrained.assign(m, 0);
    support.resize(3 * size_t(K) * n_cells);
    for (int64_t cc = 0; cc < n_cells; ++cc) {
      const int32_t* cv = &mesh.cell_vertices[4 * cc];
      for (int i = 0; i < K; ++i)
        for (int a = 0; a < 3; ++a) {
          double sum = 0;
          for (int v = 0; v < 4; ++v) {
            const int lat = p == 1 ? ref::Tables<1>::LATTICE[i][v]
                                   : p == 2 ? ref::Tables<2>::LATTICE[i][v] : ref::Tables<3>::LATTICE[i][v];
            sum += lat * mesh.x[3 * size_t(cv[v]) + a];
          }
          support[3 * (size_t(K) * cc + i) + a] = sum / p;
        }
    }
    const int n_geo = has_mass ? 11 : 10;
    std::vector<T> geo(size_t(n_geo) * n_cells);
    // per-cell quantities for the penalty
    std::vector<double> tau(n_cells), inv_h(4 * size_t(n_cells)), area(4 * size_t(n_cells));
    std::vector<double> absdet(n_cells);
    for (int64_t cc = 0; cc < n_cells; ++cc) {
      const CellGeometry g = cell_geometry(mesh, cc);
      absdet[cc] = std::fabs(g.det);
      double G[6];
      metric(g, G);
      for (int k = 0; k < 6; ++k) geo[size_t(k) * n_cells + cc] = T(G[k]);
      if (has_mass) geo[size_t(10) * n_cells + cc] = T(cfg.mass * absdet[cc]);
      double surf = 0;
      for (int f = 0; f < 4; ++f) {
        double a, nrm[3];
        face_area_normal(mesh, cc, f, a, nrm);
        area[4 * cc + f] = a;
        inv_h[4 * cc + f] = 2.0 * a / absdet[cc];  // |grad lambda_f| = 1/h_f
        surf += a * (mesh.nb[4 * cc + f] == -1 ? 1.0 : 0.5);  // -2: interior, neighbour not local
      }
      tau[cc] = surf / (absdet[cc] / 6.0);
    }
    const double factor = cfg.penalty == FEM_PENALTY_SQUARE ? double((p + 1) * (p + 1))
                                                            : double((p + 1) * (p + 3)) / 3.0;
    for (int64_t cc = 0; cc < n_cells; ++cc)
      for (int f = 0; f < 4; ++f) {
        const int32_t nbc = mesh.nb[4 * cc + f];
        double sigma;
        if (cfg.kind == FEM_HELMHOLTZ) {
          // 1/h normal to the face, averaged over both sides
          // (application_helmholtz.cc:1329-1333 and :857-859 on the boundary)
          sigma = nbc >= 0 ? factor * 0.5 * (inv_h[4 * cc + f] + inv_h[4 * size_t(nbc) + mesh.nbf[4 * cc + f]])
                           : factor * inv_h[4 * cc + f];
        } else {
          // max of the two cells' surface/volume (DG/cells_batched/application.cc:1377-1379)
          sigma = nbc >= 0 ? factor * std::max(tau[cc], tau[nbc]) : factor * tau[cc];
        }
        geo[size_t(6 + f) * n_cells + cc] = T(sigma * area[4 * cc + f]);
      }
    build_fused(mesh, geo);
    d_status.alloc(1);
    SFEM_CUDA(cudaMemset(d_status.p, 0, sizeof(int)));
    set_variant(cfg.kernel_variant);
  }

  // cells of a block of the single-launch form
  int fused_block() const {
    if (cfg.degree == 3) return cfg.n_components == 1 ? dg_fused3_cells<1>() : dg_fused3_cells<3>();
    return cfg.n_components == 1 ? dg_fused_cells<1>() : dg_fused_cells<3>();
  }

  // Geometry, outer neighbours and (P3) outer faces by blocks of cells: FusedShape
  // (P1, P2) and Fused3Shape (P3)
  struct FusedLayout {
    bool p3;
    int64_t BS;
    int NG;        // values per cell
    size_t bytes;  // of a block: the values, then four face codes per cell
  };
  FusedLayout fused_layout() const {
    FusedLayout L;
    L.p3 = cfg.degree == 3;
    L.BS = fused_block();
    L.NG = (L.p3 ? 10 : 22) + (has_mass ? 1 : 0);
    L.bytes = size_t(L.NG) * L.BS * sizeof(T) + 4 * L.BS * (L.p3 ? sizeof(uint32_t) : sizeof(uint16_t));
    return L;
  }
  void build_fused(const Mesh& mesh, const std::vector<T>& geo) {
    const FusedLayout L = fused_layout();
    const int64_t BS = L.BS, nblk = (n_cells + BS - 1) / BS;
    const bool p3 = L.p3;
    const int NG = L.NG;
    const size_t block_bytes = L.bytes;
    std::vector<unsigned char> fg(block_bytes * nblk, 0);
    std::vector<std::vector<int32_t>> outer(nblk);
    std::vector<std::vector<OuterFace<T>>> faces(p3 ? nblk : 0);
#pragma omp parallel for schedule(static)
    for (int64_t b = 0; b < nblk; ++b) {
      const int64_t c0 = b * BS, c1 = std::min(n_cells, c0 + BS);
      T* g = reinterpret_cast<T*>(fg.data() + b * block_bytes);
      uint16_t* code = reinterpret_cast<uint16_t*>(g + NG * BS);    // P1, P2
      uint32_t* code3 = reinterpret_cast<uint32_t*>(g + NG * BS);   // P3
      if (p3) std::fill(code3, code3 + 4 * BS, kBoundary3);
      else std::fill(code, code + 4 * BS, kBoundary);
      std::vector<int32_t>& ex = outer[b];
      for (int64_t cc = c0; cc < c1; ++cc)
        for (int f = 0; f < 4; ++f) {
          const int32_t nbc = mesh.nb[4 * cc + f];
          if (nbc >= 0 && (nbc < c0 || nbc >= c1)) ex.push_back(nbc);
        }
      std::sort(ex.begin(), ex.end());
      ex.erase(std::unique(ex.begin(), ex.end()), ex.end());
      for (int64_t cc = c0; cc < c1; ++cc) {
        for (int k = 0; k < 10; ++k) g[k * BS + cc - c0] = geo[size_t(k) * n_cells + cc];
        if (has_mass) g[(NG - 1) * BS + cc - c0] = geo[size_t(10) * n_cells + cc];
        for (int f = 0; f < 4; ++f) {
          const int32_t nbc = mesh.nb[4 * cc + f];
          if (nbc < 0) continue;
          const int of = mesh.nbf[4 * cc + f];
          const bool in = nbc >= c0 && nbc < c1;
          const int64_t row = in ? nbc - c0 : BS + (std::lower_bound(ex.begin(), ex.end(), nbc) - ex.begin());
          // J^-1 (2|F| n) of the neighbour on its side of the face, as the barycentric
          // weights of its three face vertices
          T w[3];
          if (!p3 || !in) {
            double G[6], c[4] = {0, 0, 0, 0};
            metric(cell_geometry(mesh, nbc), G);
            const double M[3][3] = {{G[0], G[3], G[4]}, {G[3], G[1], G[5]}, {G[4], G[5], G[2]}};
            for (int a = 0; a < 3; ++a) {
              c[a + 1] = of == 0 ? M[a][0] + M[a][1] + M[a][2] : -M[a][of - 1];
              c[0] -= c[a + 1];
            }
            for (int v = 0, k = 0; v < 4; ++v)
              if (v != of) w[k++] = T(c[v]);
          }
          if (p3) {
            uint32_t slot = 0;
            if (!in) {
              slot = uint32_t(faces[b].size());
              OuterFace<T> o;
              o.pad = T(0);
              for (int k = 0; k < 3; ++k) o.w[k] = w[k];
              o.code = uint32_t(row) | uint32_t(of) << 14;
              faces[b].push_back(o);
            }
            code3[f * BS + cc - c0] = uint32_t(row) | uint32_t(of) << 14 | slot << 16;
          } else {
            for (int k = 0; k < 3; ++k) g[(10 + 3 * f + k) * BS + cc - c0] = w[k];
            code[f * BS + cc - c0] = uint16_t(row << 2 | of);
          }
        }
      }
    }
    std::vector<int32_t> begin(nblk + 1, 0), ext, fbegin(nblk + 1, 0);
    std::vector<OuterFace<T>> all;
    for (int64_t b = 0; b < nblk; ++b) {
      n_ext = std::max(n_ext, int(outer[b].size()));
      ext.insert(ext.end(), outer[b].begin(), outer[b].end());
      begin[b + 1] = int32_t(ext.size());
      if (p3) {
        n_outer = std::max(n_outer, int(faces[b].size()));
        all.insert(all.end(), faces[b].begin(), faces[b].end());
        fbegin[b + 1] = int32_t(all.size());
      }
    }
    d_ext_begin.upload(begin);
    d_fgeo.upload(fg);
    d_ext.upload(ext);
    if (p3) {
      d_face_begin.upload(fbegin);
      d_outer.upload(all);
    }
  }

  // Geometry by cells and trace buffer, which the single-launch forms do not read
  // (Helmholtz P2 FP64: 108 and 288 of 607 bytes a cell): made when a two-launch form or
  // the diagonal is first asked for.
  std::mutex tables_mutex;
  std::atomic<bool> have_geometry{false}, have_traces{false};

  void need_geometry() {
    if (have_geometry.load(std::memory_order_acquire)) return;
    std::lock_guard<std::mutex> lock(tables_mutex);
    if (have_geometry.load(std::memory_order_relaxed)) return;
    RelaxedCapture relaxed;
    const FusedLayout L = fused_layout();
    const std::vector<unsigned char> fg = d_fgeo.download();
    const std::vector<int32_t> begin = d_ext_begin.download(), ext = d_ext.download();
    const size_t n = size_t(n_cells);
    std::vector<T> geo((has_mass ? 11 : 10) * n);
    std::vector<int32_t> nb(4 * n);
    std::vector<int8_t> nbf(4 * n);
#pragma omp parallel for schedule(static)
    for (int64_t c = 0; c < n_cells; ++c) {
      const int64_t b = c / L.BS, at = c % L.BS;
      const T* g = reinterpret_cast<const T*>(fg.data() + b * L.bytes);
      for (int k = 0; k < 10; ++k) geo[k * n + c] = g[k * L.BS + at];
      if (has_mass) geo[10 * n + c] = g[(L.NG - 1) * L.BS + at];
      const void* codes = g + L.NG * L.BS;
      for (int f = 0; f < 4; ++f) {
        const uint32_t code3 = L.p3 ? static_cast<const uint32_t*>(codes)[f * L.BS + at] : 0;
        const uint16_t code = L.p3 ? uint16_t(0) : static_cast<const uint16_t*>(codes)[f * L.BS + at];
        const bool boundary = L.p3 ? code3 == kBoundary3 : code == kBoundary;
        const int64_t row = L.p3 ? code3 & 0x3FFFu : code >> 2;
        nb[f * n + c] = boundary ? -1 : row < L.BS ? int32_t(b * L.BS + row) : ext[begin[b] + row - L.BS];
        nbf[f * n + c] = boundary ? 0 : int8_t(L.p3 ? code3 >> 14 & 3u : code & 3u);
      }
    }
    d_geo.upload(geo);
    d_nb.upload(nb);
    d_nbf.upload(nbf);
    SFEM_CUDA(cudaStreamSynchronize(nullptr));  // other streams do not wait for the copies
    have_geometry.store(true, std::memory_order_release);
  }
  size_t trace_values() const {
    return size_t((n_cells + kQB - 1) / kQB * kQB) * 4 * cfg.n_components * nfq_of(cfg.degree);
  }
  void need_traces() {
    if (have_traces.load(std::memory_order_acquire)) return;
    std::lock_guard<std::mutex> lock(tables_mutex);
    if (have_traces.load(std::memory_order_relaxed)) return;
    RelaxedCapture relaxed;
    d_Q.alloc(trace_values());
    have_traces.store(true, std::memory_order_release);
  }
  // vmult with variant v takes one launch
  bool one_launch(int v) const {
    const DGProblem<T> pr = problem(nullptr, nullptr);
    return one_launch(cfg, &pr, 1, v);
  }
  static bool one_launch(const OpConfig& cfg, const DGProblem<T>* probs, int n, int v) {
    if (v == 0) v = default_variant(cfg.degree, cfg.n_components, 0);
    if (v != 1) return false;
    return cfg.degree <= 2 || (cfg.n_components == 1 ? fused3_pays<1>(probs, n) : fused3_pays<3>(probs, n));
  }
  void set_variant(int v) override {
    if (!one_launch(v)) {
      need_geometry();
      need_traces();
    }
    cfg.kernel_variant = v;
  }

  // variant 1 in one launch or two
  std::string forms() const override {
    return one_launch(1) ? "1" : "2";
  }

  int status(bool clear) override {
    int v = 0;
    SFEM_CUDA(cudaMemcpy(&v, d_status.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (clear && v) SFEM_CUDA(cudaMemset(d_status.p, 0, sizeof(int)));
    return v;
  }

  DGProblem<T> problem(const void* src, void* dst) const {
    DGProblem<T> pr;
    pr.geo = d_geo.p;
    pr.nb = d_nb.p;
    pr.nbf = d_nbf.p;
    pr.fgeo = d_fgeo.p;
    pr.ext_begin = d_ext_begin.p;
    pr.ext = d_ext.p;
    pr.n_ext = n_ext;
    pr.face_begin = d_face_begin.p;
    pr.outer = d_outer.p;
    pr.n_outer = n_outer;
    pr.src = static_cast<const T*>(src);
    pr.dst = static_cast<T*>(dst);
    pr.Q = d_Q.p;
    pr.n_cells = n_cells;
    return pr;
  }

  void vmult(void* dst, const void* src, cudaStream_t s) override {
    const DGProblem<T> pr = problem(src, dst);
    launch_dg(cfg, &pr, 1, s, 0, d_status.p);
  }

  void vmult_phase(void* dst, const void* src, int phase, cudaStream_t s) override {
    need_geometry();
    need_traces();
    const DGProblem<T> pr = problem(src, dst);
    launch_dg(cfg, &pr, 1, s, phase, d_status.p);
  }

  size_t scratch_bytes() const override { return trace_values() * sizeof(T); }

  void vmult_with_scratch(void* dst, const void* src, void* scratch, size_t bytes, cudaStream_t s) override {
    SFEM_REQUIRE(bytes >= scratch_bytes(), FEM_ERR_ARG, "vmult: scratch too small");
    DGProblem<T> pr = problem(src, dst);
    pr.Q = static_cast<T*>(scratch);
    launch_dg(cfg, &pr, 1, s, 0, d_status.p);
  }

  void diagonal(void* diag, cudaStream_t s) override {
    need_geometry();
    const DGProblem<T> pr = problem(nullptr, diag);
    launch_dg(cfg, &pr, 1, s, 3, d_status.p);
  }

  void work(double& flops, double& bytes) const override {
    const int p = cfg.degree, kq = kq_of(p), nf = nf_of(p), nfq = nfq_of(p), nz = nnz_grad_rt(p);
    const double trace = 2.0 * (nz + 12 * nfq);
    double apply = 2.0 * (2 * nz + 9 * kq + 3 * kq * kq) +
                   4 * 2.0 * (3 * nfq + nf + nf * nf + nf + 2 * nf * nfq + 3 * nfq + 3 * nfq);
    if (has_mass) apply += 2.0 * (K * K + K);
    flops = (trace + apply) * cfg.n_components * double(n_cells);
    const double s = double(sizeof(T));
    bytes = 2 * s * double(m) + 6 * s * double(n_cells) + double(n_interior_faces) * (8 + s) +
            double(n_boundary_faces) * (4 + s);
  }

  // Dispatch over n problems.  what: 0 trace+apply, 1 trace, 2 apply, 3 diagonal.
  // status: device word set by the bounded waits of the bulk-copy trace pass.
  static void launch_dg(const OpConfig& cfg, const DGProblem<T>* probs, int n, cudaStream_t s, int what,
                        int* status) {
    const bool mass = cfg.kind == FEM_HELMHOLTZ;
    const int nc = cfg.n_components;
    SFEM_REQUIRE(nc == 1 || nc == 3, FEM_ERR_ARG, "DG: n_components must be 1 or 3");
    SFEM_REQUIRE(n >= 1 && n <= kMaxBatch, FEM_ERR_ARG, "DG: 1..40 problems per launch");
    const int variant = cfg.kernel_variant > 0 ? cfg.kernel_variant : default_variant(cfg.degree, nc, what);
#define SFEM_DG_CASE(P, NC, MASS)                                                       \
  if (cfg.degree == P && nc == NC && mass == MASS) {                                    \
    run<P, NC, MASS>(probs, n, s, what, variant, status);                               \
    return;                                                                             \
  }
    SFEM_DG_CASE(1, 1, false) SFEM_DG_CASE(2, 1, false) SFEM_DG_CASE(3, 1, false)
    SFEM_DG_CASE(1, 1, true) SFEM_DG_CASE(2, 1, true) SFEM_DG_CASE(3, 1, true)
    SFEM_DG_CASE(1, 3, true) SFEM_DG_CASE(2, 3, true) SFEM_DG_CASE(3, 3, true)
    SFEM_DG_CASE(1, 3, false) SFEM_DG_CASE(2, 3, false) SFEM_DG_CASE(3, 3, false)
#undef SFEM_DG_CASE
    throw Error(FEM_ERR_ARG, "DG: unsupported degree/components combination");
  }

  // kernel forms: 1 one launch with a thread per cell and component, its single
  // phases with 128 cells per CTA; 2 thread per cell, 64 cells per CTA; 3 warp
  // roles, 32 cells per CTA.  Single phases (vmult_phase) of scalar FP32 P3 run
  // best with the results in registers and 8 CTAs per SM (B200, 32^3: 38 us for
  // both against 44).
  static int default_variant(int p, int nc, int what) { return (nc == 1 && p == 3 && sizeof(T) == 4 && what != 0) ? 4 : 1; }

  static DGBatch<T> make_batch(const DGProblem<T>* probs, int n, int bs, int64_t& n_blocks) {
    DGBatch<T> b;
    b.n = n;
    b.block_begin[0] = 0;
    for (int i = 0; i < n; ++i) {
      b.p[i] = probs[i];
      b.block_begin[i + 1] = b.block_begin[i] + (probs[i].n_cells + bs - 1) / bs;
    }
    n_blocks = b.block_begin[n];
    return b;
  }

  template <class K>
  static void opt_in_smem(K kernel, size_t bytes, std::atomic<uint64_t>& configured) {
    int dev = 0;
    SFEM_CUDA(cudaGetDevice(&dev));
    once_per_device(configured, dev, [&] {
      SFEM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
    });
  }

  // The bulk-copy trace pass needs every copy 16-byte aligned and a whole
  // number of 16-byte units: src rows (the last block's included) and the
  // metric rows of the geometry.
  template <int P>
  static bool trace_tma_ok(const DGProblem<T>* probs, int n) {
    for (int i = 0; i < n; ++i) {
      const DGProblem<T>& pr = probs[i];
      if ((reinterpret_cast<uintptr_t>(pr.src) | reinterpret_cast<uintptr_t>(pr.geo)) & 15u) return false;
      if ((size_t(pr.n_cells) * sizeof(T)) % 16 != 0) return false;  // metric row starts
      if ((size_t(pr.n_cells % kQB) * k_of(P) * sizeof(T)) % 16 != 0) return false;
    }
    return true;
  }
  template <int P>
  static void run_trace_tma(const DGBatch<T>& b, int64_t n_blocks, cudaStream_t s, int* status) {
    constexpr int NS = 3;
    using S = TraceTmaShape<T, gen::Ops<P>::K, NS>;
    auto kern = dg_trace_tma_kernel<P, T, NS>;
    static std::atomic<uint64_t> conf{0};
    static int grid_per_dev[64] = {};
    int dev = 0;
    SFEM_CUDA(cudaGetDevice(&dev));
    once_per_device(conf, dev, [&] {
      SFEM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
      int sms = 0, occ = 0;
      SFEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      SFEM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kQB, S::SMEM));
      SFEM_REQUIRE(occ > 0, FEM_ERR_CUDA, "DG trace pass does not fit on an SM");
      grid_per_dev[dev] = sms * occ;
    });
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(n_blocks, grid_per_dev[dev]));
    launch_pdl(kern, unsigned(grid), kQB, S::SMEM, s, b, n_blocks, status);
  }

  // PDLM > 0 (scalar problems): the apply pass is launched as a programmatic
  // dependent of the trace pass (see dg_apply_kernel)
  template <int P, int NC, bool MASS, int BS, int MINB = (BS == 64 ? 6 : 1), bool ALIAS = false, int PDLM = 0>
  static void run_cell(const DGProblem<T>* probs, int n, cudaStream_t s, int what, int* status) {
    using S = DGShape<P, NC>;
    int64_t n_blocks = 0;
    const DGBatch<T> b = make_batch(probs, n, BS, n_blocks);
    const size_t sm_trace = size_t(BS) * (S::US + S::QS) * sizeof(T);
    // scalar problems: block-major traces (no shared memory in the trace pass)
    constexpr bool BQ = NC == 1;
    const size_t sm_apply = size_t(BS) * ((ALIAS ? 1 : 2) * S::US + S::QS) * sizeof(T);
    static std::atomic<uint64_t> conf_t{0}, conf_a{0};
    auto apply = dg_apply_kernel<P, NC, MASS, BS, T, MINB, ALIAS, BQ, (BQ ? PDLM : 0)>;
    opt_in_smem(apply, sm_apply, conf_a);
    if (what != 2) {
      if constexpr (BQ) {
        int64_t nbt = 0;
        const DGBatch<T> bt = make_batch(probs, n, kQB, nbt);
        if (trace_tma_ok<P>(probs, n)) run_trace_tma<P>(bt, nbt, s, status);
        else launch_pdl(dg_trace_blk_kernel<P, T>, unsigned(nbt), kQB, 0, s, bt, nbt);
      } else {
        opt_in_smem(dg_trace_kernel<P, NC, BS, T>, sm_trace, conf_t);
        dg_trace_kernel<P, NC, BS, T><<<unsigned(n_blocks), BS, sm_trace, s>>>(b, n_blocks);
      }
    }
    if (what == 1) return;
    if (BQ && PDLM > 0 && what == 0) {
      // the trace pass just launched on this stream is the only producer the
      // apply pass may overlap: everything else it reads was complete before
      // the trace pass started
      launch_pdl(apply, unsigned(n_blocks), BS, sm_apply, s, b, n_blocks);
    } else {
      apply<<<unsigned(n_blocks), BS, sm_apply, s>>>(b, n_blocks);
    }
  }

  // P1 and P2 in one pass (kernels_dg_fused.cuh)
  template <int P, int NC, bool MASS>
  static void run_fused(const DGProblem<T>* probs, int n, cudaStream_t s) {
    constexpr int BS = dg_fused_cells<NC>();
    using S = FusedShape<P, NC, MASS, BS, T>;
    int64_t n_blocks = 0;
    const DGBatch<T> b = make_batch(probs, n, BS, n_blocks);
    int rows = BS;
    for (int i = 0; i < n; ++i) rows = std::max(rows, BS + probs[i].n_ext);
    static std::atomic<uint64_t> conf{0};
    auto kern = dg_fused_kernel<P, NC, MASS, BS, T, dg_fused_min_ctas<P, NC, T>()>;
    // at most BS cells with four outer neighbours each
    opt_in_smem(kern, S::bytes(5 * BS), conf);
    launch_pdl(kern, unsigned(n_blocks), BS * NC, S::bytes(rows), s, b, rows);
  }

  // P3 in one launch pays except for scalar FP64 with most neighbours outside
  // the block, where a CTA's shared memory holds five rows per cell and one CTA
  // fits an SM (B200, DG P3, 24^3 hexes, us per vmult, one launch / two): cells by
  // x-rows (1.3 outer faces per cell) FP64 22.4 / 29.5, FP32 14.4 / 18.3; cells in
  // random order (4) FP64 45.4 / 38.4, FP32 26.6 / 44.7; 3 components FP64 168 /
  // 186, FP32 65 / 117.  The FP64 lines through both points meet near 2.7.
  template <int NC>
  static bool fused3_pays(const DGProblem<T>* probs, int n) {
    if (NC > 1 || sizeof(T) == 4) return true;
    for (int i = 0; i < n; ++i)
      if (probs[i].n_outer > 5 * dg_fused3_cells<NC>() / 2) return false;
    return true;
  }

  // P3 in one launch (kernels_dg_fused3.cuh)
  template <int NC, bool MASS>
  static void run_fused3(const DGProblem<T>* probs, int n, cudaStream_t s) {
    constexpr int BS = dg_fused3_cells<NC>();
    using S = Fused3Shape<NC, MASS, BS, T>;
    int64_t n_blocks = 0;
    const DGBatch<T> b = make_batch(probs, n, BS, n_blocks);
    int ne = 0, nf = 0;
    for (int i = 0; i < n; ++i) {
      ne = std::max(ne, probs[i].n_ext);
      nf = std::max(nf, probs[i].n_outer);
    }
    static std::atomic<uint64_t> conf{0};
    auto kern = dg_fused3_kernel<NC, MASS, BS, T, dg_fused3_min_ctas<NC, T>()>;
    // at most BS cells with four outer neighbours each
    opt_in_smem(kern, S::bytes(4 * BS, 4 * BS), conf);
    launch_pdl(kern, unsigned(n_blocks), BS * NC, S::bytes(ne, nf), s, b, ne, nf);
  }

  // trace + apply with the cross-block neighbour data prefetched (scalar problems)
  template <int P, int BS, int XCAP>
  static void run_xp(const DGProblem<T>* probs, int n, cudaStream_t s, int what) {
    using S = DGShape<P, 1>;
    using O = gen::Ops<P>;
    int64_t n_blocks = 0;
    const DGBatch<T> b = make_batch(probs, n, BS, n_blocks);
    const size_t sm_trace = size_t(BS) * (S::US + S::QS) * sizeof(T);
    const size_t sm_apply = (size_t(BS) * (2 * S::US + S::QS) + size_t(XCAP) * (O::NF + O::NFQ)) * sizeof(T);
    static std::atomic<uint64_t> conf_t{0}, conf_a{0};
    auto trace = dg_trace_kernel<P, 1, BS, T>;
    auto apply = dg_apply_xp_kernel<P, BS, XCAP, T>;
    opt_in_smem(trace, sm_trace, conf_t);
    opt_in_smem(apply, sm_apply, conf_a);
    if (what != 2) trace<<<unsigned(n_blocks), BS, sm_trace, s>>>(b, n_blocks);
    if (what != 1) apply<<<unsigned(n_blocks), BS, sm_apply, s>>>(b, n_blocks);
  }

  // phase-split scalar kernels (kernels_dg2.cuh): cross-block trace + apply
  template <int P, bool MASS, int BS, int MINB, bool YS = false>
  static void run_split(const DGProblem<T>* probs, int n, cudaStream_t s, int what) {
    using S = DG2Shape<P, YS>;
    int64_t n_blocks = 0;
    const DGBatch<T> b = make_batch(probs, n, BS, n_blocks);
    const size_t sm_trace = size_t(BS) * S::US * sizeof(T);
    const size_t sm_apply = size_t(BS) * S::ELEMS * sizeof(T);
    static std::atomic<uint64_t> conf_t{0}, conf_a{0};
    auto trace = dg_trace_cross_kernel<P, BS, T>;
    auto apply = dg_apply2_kernel<P, MASS, BS, T, MINB, YS>;
    opt_in_smem(trace, sm_trace, conf_t);
    opt_in_smem(apply, sm_apply, conf_a);
    if (what != 2) trace<<<unsigned(n_blocks), BS, sm_trace, s>>>(b, n_blocks);
    if (what != 1) apply<<<unsigned(n_blocks), BS, sm_apply, s>>>(b, n_blocks);
  }

  template <int P, int NC, bool MASS>
  static void run_warp(const DGProblem<T>* probs, int n, cudaStream_t s, int what) {
    using D = DG3<P, NC>;
    int64_t n_blocks = 0;
    const DGBatch<T> b = make_batch(probs, n, D::CELLS, n_blocks);
    const size_t sm_trace = size_t(D::TRACE_ELEMS) * sizeof(T);
    const size_t sm_apply = size_t(D::APPLY_ELEMS) * sizeof(T);
    static std::atomic<uint64_t> conf_t{0}, conf_a{0};
    opt_in_smem(dg3_trace_kernel<P, NC, T>, sm_trace, conf_t);
    opt_in_smem(dg3_apply_kernel<P, NC, MASS, T>, sm_apply, conf_a);
    if (what != 2) dg3_trace_kernel<P, NC, T><<<unsigned(n_blocks), D::THREADS, sm_trace, s>>>(b, n_blocks);
    if (what != 1) dg3_apply_kernel<P, NC, MASS, T><<<unsigned(n_blocks), D::THREADS, sm_apply, s>>>(b, n_blocks);
  }

  template <int P, int NC, bool MASS>
  static void run(const DGProblem<T>* probs, int n, cudaStream_t s, int what, int variant, int* status) {
    if (what == 3) {
      int64_t n_blocks = 0;
      const DGBatch<T> b = make_batch(probs, n, 128, n_blocks);
      dg_diagonal_kernel<P, NC, MASS, T><<<unsigned(n_blocks), 128, 0, s>>>(b, n_blocks);
    } else if (variant == 1 && P <= 2 && what == 0) {
      // P1 and P2: one pass (B200, 45 x 38 x 31 hexes: see kernels_dg_fused.cuh); the
      // two passes below are what vmult_phase runs
      if constexpr (P <= 2) run_fused<P, NC, MASS>(probs, n, s);
    } else if (variant == 1 && what == 0 && fused3_pays<NC>(probs, n)) {
      if constexpr (P == 3) run_fused3<NC, MASS>(probs, n, s);
    } else if (variant == 1) {
      // scalar problems: the apply pass loads its geometry and src rows while
      // the trace pass finishes (B200, DG P3 FP64 32^3: 68.5 -> 64.5 us per vmult)
      run_cell<P, NC, MASS, 128, 1, false, 1>(probs, n, s, what, status);
    } else if (variant == 2) {
      run_cell<P, NC, MASS, 64>(probs, n, s, what, status);
    } else if (variant == 3) {
      run_warp<P, NC, MASS>(probs, n, s, what);
    } else if (variant == 5) {
      // 64 cells per CTA, 5 CTAs per SM (up to 204 registers: no spills for P3)
      run_cell<P, NC, MASS, 64, 5, false>(probs, n, s, what, status);
    } else if (variant == 4) {
      // 64 cells per CTA, results aliased onto the staged src rows (scalar
      // problems), registers capped for 8 CTAs per SM; for scalar problems the
      // cell term is computed while the trace pass finishes (B200, DG P3 FP32
      // 32^3: 41.8 -> 38.0 us per vmult)
      if (NC == 1) run_cell<P, NC, MASS, 64, 8, (NC == 1), 2>(probs, n, s, what, status);
      else run_cell<P, NC, MASS, 64, 8, false>(probs, n, s, what, status);
    } else if (variant == 7 || variant == 9) {
      // phase-split scalar kernels (kernels_dg2.cuh): 7 results in registers,
      // 64 cells x 5 CTAs per SM; 9 results in shared memory, 64 cells x 4
      // CTAs (no spills); multi-component problems take the 128-cell form
      if constexpr (NC == 1) {
        if (variant == 7) run_split<P, MASS, 64, 5>(probs, n, s, what);
        else run_split<P, MASS, 64, 4, true>(probs, n, s, what);
      } else {
        run_cell<P, NC, MASS, 128>(probs, n, s, what, status);
      }
    } else if (variant == 11) {
      // 128 cells per CTA with the cross-block neighbour data prefetched into
      // shared memory; multi-component and mass problems take the 128-cell form
      if constexpr (NC == 1 && !MASS) run_xp<P, 128, 192>(probs, n, s, what);
      else run_cell<P, NC, MASS, 128>(probs, n, s, what, status);
    } else {
      throw Error(FEM_ERR_ARG, "DG: kernel variant must be 0..5, 7, 9 or 11");
    }
    SFEM_CUDA(cudaGetLastError());
  }
};

template <typename T>
class DGBatchImpl final : public Batch {
 public:
  std::vector<DGOperator<T>*> ops;
  // an operator listed more than once (several right-hand sides on one mesh)
  // gets a trace scratch of its own for every repeat: the two passes of one
  // launch must not share it between problems
  std::vector<DevBuf<T>> extra_q;
  std::vector<int> q_of;  // -1: the operator's own scratch, else index into extra_q
  OpConfig cfg;
  explicit DGBatchImpl(const std::vector<Operator*>& o) {
    SFEM_REQUIRE(!o.empty() && int(o.size()) <= kMaxBatch, FEM_ERR_ARG, "batch: 1..40 operators");
    cfg = o[0]->cfg;
    for (auto* op : o) {
      auto* d = dynamic_cast<DGOperator<T>*>(op);
      SFEM_REQUIRE(d != nullptr, FEM_ERR_ARG, "batch: only DG/Helmholtz operators of one precision");
      SFEM_REQUIRE(d->cfg.degree == cfg.degree && d->cfg.kind == cfg.kind &&
                       d->cfg.n_components == cfg.n_components,
                   FEM_ERR_ARG, "batch: operators must share kind, degree and components");
      int repeat = -1;
      for (auto* prev : ops)
        if (prev == d) repeat = 0;
      if (repeat == 0) {
        extra_q.emplace_back(d->scratch_bytes() / sizeof(T));
        repeat = int(extra_q.size()) - 1;
      }
      q_of.push_back(repeat);
      ops.push_back(d);
    }
    set_variant(cfg.kernel_variant);
  }
  void vmult(void* const* dst, const void* const* src, cudaStream_t s) override {
    DGProblem<T> probs[kMaxBatch];
    for (size_t i = 0; i < ops.size(); ++i) {
      probs[i] = ops[i]->problem(src[i], dst[i]);
      if (q_of[i] >= 0) probs[i].Q = extra_q[q_of[i]].p;
    }
    DGOperator<T>::launch_dg(cfg, probs, int(ops.size()), s, 0, ops[0]->d_status.p);
  }
  int variant() const override { return cfg.kernel_variant; }
  void set_variant(int v) override {
    SFEM_REQUIRE(v >= 0 && v <= 11 && v != 6 && v != 8 && v != 10, FEM_ERR_ARG,
                 "batch: kernel variant must be 0..5, 7, 9 or 11");
    DGProblem<T> probs[kMaxBatch];
    for (size_t i = 0; i < ops.size(); ++i) probs[i] = ops[i]->problem(nullptr, nullptr);
    if (!DGOperator<T>::one_launch(cfg, probs, int(ops.size()), v))
      for (auto* o : ops) {
        o->need_geometry();
        o->need_traces();
      }
    cfg.kernel_variant = v;
  }
  TuneResult tune(int reps, bool use_cache) override {
    TuneResult res;
    res.us.assign(5, 0.0);
    int64_t cells = 0;
    std::string forms = "1";
    for (auto* o : ops) {
      cells += o->n_cells;
      forms = std::max(forms, o->forms());  // one problem can send the launch to two
    }
    const std::vector<int> cand = tune_candidates(cfg);
    const std::string key = "batch" + std::to_string(ops.size()) + "," + tune_key(cfg, cells, forms);
    if (use_cache) {
      const int v = tune_lookup(key);
      if (std::find(cand.begin(), cand.end(), v) != cand.end()) {
        set_variant(v);
        res.variant = v;
        res.cached = true;
        return res;
      }
    }
    std::vector<DevBuf<T>> bufs;
    std::vector<void*> d(ops.size());
    std::vector<const void*> x(ops.size());
    for (size_t i = 0; i < ops.size(); ++i) {
      bufs.emplace_back(size_t(ops[i]->m));
      bufs.emplace_back(size_t(ops[i]->m));
      SFEM_CUDA(cudaMemset(bufs[2 * i].p, 0, sizeof(T) * ops[i]->m));
    }
    for (size_t i = 0; i < ops.size(); ++i) {
      x[i] = bufs[2 * i].p;
      d[i] = bufs[2 * i + 1].p;
    }
    cudaStream_t s = nullptr;
    SFEM_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    const int keep = cfg.kernel_variant;
    double best = 1e300;
    try {
      for (int v : cand) {
        set_variant(v);
        const double us = time_launches([&](cudaStream_t st) { vmult(d.data(), x.data(), st); }, reps, s);
        res.us[v - 1] = us;
        if (us < best) {
          best = us;
          res.variant = v;
        }
      }
    } catch (...) {
      cfg.kernel_variant = keep;
      cudaStreamDestroy(s);
      throw;
    }
    cudaStreamDestroy(s);
    cfg.kernel_variant = res.variant;
    tune_store(key, res.variant, res.us);
    return res;
  }
};

}  // namespace

template <typename T>
std::unique_ptr<Operator> make_dg_operator(const Mesh& mesh, const OpConfig& cfg) {
  return std::make_unique<DGOperator<T>>(mesh, cfg);
}
template <typename T>
std::unique_ptr<Batch> make_dg_batch(const std::vector<Operator*>& ops) {
  return std::make_unique<DGBatchImpl<T>>(ops);
}

}  // namespace sfem
