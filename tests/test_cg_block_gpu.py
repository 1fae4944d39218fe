"""Block form of the CG operators (4 x 4 x 4 hexes per step) at the edges of its
range: sides that 4 does not divide, boxes thinner than a block, one block, more
blocks than resident CTAs, partitions and three components; against the oracle."""
import numpy as np
import pytest

import oracle as orc
import simplexfem as sf
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu

# FP64: the repository's 1e-12; FP32: 2e-6 (tests of the other forms)
TOL = {"fp64": 1e-12, "fp32": 2e-6}


def product(op, x):
    import torch
    src = torch.tensor(x, dtype=op.dtype, device="cuda")
    dst = torch.full_like(src, float("nan"))
    op.vmult(dst, src)
    return dst.double().cpu().numpy(), src.double().cpu().numpy()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n", [(4, 4, 4), (5, 3, 9), (1, 13, 2), (12, 8, 4), (21, 18, 23)])
def test_block_form_matches_oracle(cuda, n, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=5)
    op = sf.Operator(mesh, p, "cg", precision)
    op.set_kernel_variant(3)
    y, x = product(op, seeded_src(op.m(), 3))
    ref = orc.for_mesh(mesh, p, orc.CG).vmult(x)
    assert rel_l2(y, ref) <= TOL[precision]


@pytest.mark.parametrize("p, precision, tol", [(1, "fp64", 1e-13), (2, "fp64", 1e-13), (3, "fp32", 2e-6)])
def test_block_form_many_blocks_per_cta(cuda, p, precision, tol):
    """Blocks beyond the persistent grid: the forms of the operator agree."""
    mesh = sf.Mesh((50, 46, 54), jitter=0.1, seed=1)
    op = sf.Operator(mesh, p, "cg", precision)
    x = seeded_src(op.m(), 9)
    op.set_kernel_variant(1)
    ref, _ = product(op, x)
    op.set_kernel_variant(3)
    y, _ = product(op, x)
    assert rel_l2(y, ref) <= tol


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n", [(24, 24, 24), (23, 26, 25)])
def test_three_component_block_form(cuda, n, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=5)
    op = sf.Operator(mesh, p, "cg", precision, n_components=3)
    y, x = product(op, seeded_src(op.m(), 3))
    o = orc.for_mesh(mesh, p, orc.CG)
    for k in range(3):
        assert rel_l2(y[k::3], o.vmult(np.ascontiguousarray(x[k::3]))) <= TOL[precision]
