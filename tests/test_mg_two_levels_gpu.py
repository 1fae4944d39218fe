"""The coarse correction of a two-level hierarchy, whose products on level 0 come before
any other: a small host program against the library's C++ interface, since no entry
point of the C ABI reaches it with fewer than three levels."""
import os
import subprocess

import pytest

import simplexfem as sf

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "mesh.hpp"
#include "mg.hpp"
using namespace sfem;
int main() {
  MeshDescription d;
  d.n[0] = d.n[1] = d.n[2] = 4;
  for (int a = 0; a < 3; ++a) { d.lo[a] = 0; d.hi[a] = 1; }
  d.jitter = 0; d.seed = 0;
  const Mesh mesh = build_kuhn_mesh(d);
  OpConfig cfg;  // CG P2 FP64
  auto op = make_operator(mesh, cfg);
  MGParams p;
  p.precision = FEM_FP64;
  p.coarse_n = 4;
  // what the hierarchy's vectors are allocated from is full of NaNs
  std::vector<void*> junk;
  for (size_t bytes : {size_t(1) << 10, size_t(2) << 10, size_t(8) << 10, size_t(1) << 20, size_t(16) << 20})
    for (int k = 0; k < 64; ++k) {
      void* q = nullptr;
      if (cudaMalloc(&q, bytes) != cudaSuccess) return 2;
      cudaMemset(q, 0xFF, bytes);
      junk.push_back(q);
    }
  cudaDeviceSynchronize();
  for (void* q : junk) cudaFree(q);
  auto mg = make_multigrid(*op, p);
  if (mg->n_levels() != 2) return 3;
  DevBuf<double> r(op->m), x(op->m);
  std::vector<double> h(op->m);
  for (int64_t i = 0; i < op->m; ++i) h[i] = op->constrained[i] ? 0.0 : std::sin(double(i));
  r.upload(h);
  std::vector<double> a(op->m), b(op->m);
  for (std::vector<double>* out : {&a, &b}) {
    mg->coarse_correction(r.p, x.p, 2, nullptr);
    cudaDeviceSynchronize();
    cudaMemcpy(out->data(), x.p, sizeof(double) * op->m, cudaMemcpyDeviceToHost);
  }
  double n = 0, e = 0;
  for (int64_t i = 0; i < op->m; ++i) { n += a[i] * a[i]; e += (a[i] - b[i]) * (a[i] - b[i]); }
  std::printf("norm %.17g difference %.17g\n", std::sqrt(n), std::sqrt(e));
  return std::isfinite(n) && n > 0 && e <= 1e-24 * n ? 0 : 1;
}
"""


def test_coarse_correction_of_two_levels(cuda, tmp_path):
    src, exe = tmp_path / "two.cpp", tmp_path / "two"
    src.write_text(PROGRAM)
    pkg = os.path.dirname(sf.LIB_PATH)
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run([os.path.join(home, "bin", "nvcc"), "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(pkg, "csrc"), str(src), "-o", str(exe), sf.LIB_PATH, "-Xlinker",
                    "-rpath," + pkg], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, (run.returncode, run.stdout, run.stderr)
