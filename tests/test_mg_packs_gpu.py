"""Chebyshev smoothing of large levels, 16 bytes at once: vectors at 16-byte addresses
against the same vectors one value off, which go value by value."""
import pytest

import simplexfem as sf

pytestmark = pytest.mark.gpu


# FP32: the sums of the operator's atomics come in any order; FP64 likewise
@pytest.mark.parametrize("precision, n, tol", [("fp32", 48, 2e-6), ("fp64", 36, 1e-14)])
@pytest.mark.parametrize("zero_initial", [True, False])
def test_aligned_and_offset_vectors_agree(cuda, precision, n, tol, zero_initial):
    import torch
    op = sf.Operator(sf.Mesh((n, n, n), jitter=0.1, seed=3), 3, "cg", "fp64")
    mg = sf.Multigrid(op, precision=precision, coarse_n=3 if n == 48 else 9)
    level = mg.n_levels - 1
    m = mg.level_info(level)["m"]
    dt = mg.level_vector(level).dtype
    assert m % 2 == 1  # a last, partial pack
    gen = torch.Generator("cuda").manual_seed(5)
    b, x0 = (torch.rand(m, dtype=dt, device="cuda", generator=gen) - 0.5 for _ in range(2))
    out = []
    for off in (0, 1):
        bv, xv = (torch.empty(m + off, dtype=dt, device="cuda")[off:] for _ in range(2))
        bv.copy_(b)
        xv.copy_(x0)
        mg.smooth(level, xv, bv, zero_initial)
        out.append(xv.clone())
    assert ((out[0] - out[1]).norm() / out[0].norm()).item() <= tol
