// Host helpers shared by the operator classes: space dimensions, launch grids
// and the affine metric.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "common.hpp"
#include "mesh.hpp"
#include "ref_tables.h"

namespace sfem {
inline unsigned blocks_for(int64_t n, int bs) { return unsigned((n + bs - 1) / bs); }

// Lets this thread allocate and copy while one of its streams is being captured.
class RelaxedCapture {
 public:
  RelaxedCapture() { SFEM_CUDA(cudaThreadExchangeStreamCaptureMode(&mode_)); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  RelaxedCapture(const RelaxedCapture&) = delete;
  RelaxedCapture& operator=(const RelaxedCapture&) = delete;

 private:
  cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

template <int P>
inline int nnz_grad() {
  int z = 0;
  using Tb = ref::Tables<P>;
  for (int a = 0; a < 3; ++a)
    for (int m = 0; m < Tb::KQ; ++m)
      for (int i = 0; i < Tb::K; ++i) z += Tb::D[a][m][i] != 0.0;
  return z;
}
inline int nnz_grad_rt(int p) { return p == 1 ? nnz_grad<1>() : p == 2 ? nnz_grad<2>() : nnz_grad<3>(); }
inline int kq_of(int p) { return p == 1 ? 1 : p == 2 ? 4 : 10; }
inline int k_of(int p) { return (p + 1) * (p + 2) * (p + 3) / 6; }
inline int nf_of(int p) { return (p + 1) * (p + 2) / 2; }
inline int nfq_of(int p) { return p == 1 ? 1 : p * (p + 1) / 2; }

// metric G = |det J| J^-1 J^-T as (00,11,22,01,02,12)
inline void metric(const CellGeometry& g, double G[6]) {
  const double ad = std::fabs(g.det);
  auto mm = [&](int a, int b) {
    double s = 0;
    for (int c = 0; c < 3; ++c) s += g.Jinv[a][c] * g.Jinv[b][c];
    return ad * s;
  };
  G[0] = mm(0, 0); G[1] = mm(1, 1); G[2] = mm(2, 2);
  G[3] = mm(0, 1); G[4] = mm(0, 2); G[5] = mm(1, 2);
}

}  // namespace sfem
