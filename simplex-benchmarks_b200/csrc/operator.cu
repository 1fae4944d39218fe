// Operators: factories over kinds and precisions, inverse diagonal, CSR product.
#include <cmath>

#include "kernels_cg.cuh"
#include "op_shapes.hpp"
#include "operator.hpp"
#include "operator_parts.hpp"

namespace sfem {

namespace {

template <typename T>
__global__ void inverse_diagonal_kernel(int64_t n, T* d) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) {
    const T v = d[i];
    d[i] = fabs(double(v)) > 1e-10 ? T(1) / v : T(1);
  }
}

}  // namespace


void Operator::inverse_diagonal(void* diag, cudaStream_t s) {
  diagonal(diag, s);
  const unsigned grid = blocks_for(m, 256);
  if (cfg.precision == FEM_FP64)
    inverse_diagonal_kernel<double><<<grid, 256, 0, s>>>(m, static_cast<double*>(diag));
  else
    inverse_diagonal_kernel<float><<<grid, 256, 0, s>>>(m, static_cast<float*>(diag));
  SFEM_CUDA(cudaGetLastError());
}

std::unique_ptr<Operator> make_operator(const Mesh& mesh, const OpConfig& cfg) {
  SFEM_REQUIRE(cfg.degree >= 1 && cfg.degree <= 3, FEM_ERR_ARG, "operator: degree must be 1, 2 or 3");
  SFEM_REQUIRE(cfg.precision == FEM_FP64 || cfg.precision == FEM_FP32, FEM_ERR_ARG, "operator: bad precision");
  std::unique_ptr<Operator> op;
  if (mesh.curved) {
    SFEM_REQUIRE(cfg.kind == FEM_CG, FEM_ERR_ARG,
                 "curved meshes: CG operators only (the DG face terms are affine in this library)");
    op = make_curved_cg_operator(mesh, cfg);
  } else if (cfg.kind == FEM_CG) {
    SFEM_REQUIRE(cfg.n_components == 1 || cfg.n_components == 3, FEM_ERR_ARG, "CG: n_components must be 1 or 3");
    if (cfg.n_components == 3) {
      SFEM_REQUIRE(!cfg.weak_bc && (cfg.kernel_variant == 0 || cfg.kernel_variant == 1), FEM_ERR_ARG,
                   "CG with 3 components: strong constraints and the cell kernel only");
    }
    op = cfg.precision == FEM_FP64 ? make_cg_operator<double>(mesh, cfg) : make_cg_operator<float>(mesh, cfg);
  } else if (cfg.kind == FEM_DG || cfg.kind == FEM_HELMHOLTZ) {
    op = cfg.precision == FEM_FP64 ? make_dg_operator<double>(mesh, cfg) : make_dg_operator<float>(mesh, cfg);
  } else {
    throw Error(FEM_ERR_ARG, "operator: unknown kind");
  }
  op->mesh = &mesh;
  return op;
}

void csr_spmv(int64_t n_rows, const int64_t* row_ptr, const int32_t* col, const void* val, const void* x, void* y,
              int precision, cudaStream_t s) {
  constexpr int LANES = 8;
  const unsigned grid = blocks_for(std::max<int64_t>(n_rows, 1) * LANES, 256);
  if (precision == FEM_FP64)
    csr_spmv_kernel<double, LANES><<<grid, 256, 0, s>>>(n_rows, row_ptr, col, static_cast<const double*>(val),
                                                        static_cast<const double*>(x), static_cast<double*>(y));
  else
    csr_spmv_kernel<float, LANES><<<grid, 256, 0, s>>>(n_rows, row_ptr, col, static_cast<const float*>(val),
                                                       static_cast<const float*>(x), static_cast<float*>(y));
  SFEM_CUDA(cudaGetLastError());
}

std::unique_ptr<Operator> make_local_operator(std::shared_ptr<const Mesh> mesh, const CGDofs* dofs,
                                              const std::vector<uint8_t>* identity, const OpConfig& cfg) {
  SFEM_REQUIRE(cfg.degree >= 1 && cfg.degree <= 3, FEM_ERR_ARG, "operator: degree must be 1, 2 or 3");
  SFEM_REQUIRE(cfg.precision == FEM_FP64 || cfg.precision == FEM_FP32, FEM_ERR_ARG, "operator: bad precision");
  std::unique_ptr<Operator> op;
  if (cfg.kind == FEM_CG) {
    SFEM_REQUIRE(dofs && identity, FEM_ERR_INTERNAL, "CG local operator needs its numbering");
    op = cfg.precision == FEM_FP64 ? make_cg_local_operator<double>(*mesh, *dofs, identity, cfg)
                                   : make_cg_local_operator<float>(*mesh, *dofs, identity, cfg);
  } else {
    op = make_operator(*mesh, cfg);
  }
  op->mesh = mesh.get();
  op->owned_mesh = std::move(mesh);
  return op;
}

std::unique_ptr<Batch> make_batch(const std::vector<Operator*>& ops) {
  SFEM_REQUIRE(!ops.empty(), FEM_ERR_ARG, "batch: empty");
  return ops[0]->cfg.precision == FEM_FP64 ? make_dg_batch<double>(ops) : make_dg_batch<float>(ops);
}

}  // namespace sfem