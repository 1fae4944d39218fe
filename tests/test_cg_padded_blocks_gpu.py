"""Padded blocks (sides that 4 does not divide) where the block form had been tried on
few of them: weak boundary terms (no constrained DoFs, so the nodes of absent hexes'
sides carry values), by blocks and by patches, three components on thin boxes and on
a single block; against the oracle."""
import numpy as np
import pytest

import oracle as orc
import simplexfem as sf
from test_cg_block_gpu import TOL, product
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


def weak_oracle(mesh, p):
    dofs, fixed = mesh.cg_dofs(p)
    return orc.Oracle(mesh.vertices(), mesh.cells(), p, orc.CG, cell_dofs=dofs, constrained=fixed, weak_bc=True)


# 216 padded blocks and a few, asked for; by default P1 216 blocks, P2 and P3 patches
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n, variant", [((21, 22, 23), 3), ((5, 3, 9), 3), ((21, 22, 23), 0)])
def test_weak_boundary(cuda, n, variant, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=5)
    op = sf.Operator(mesh, p, "cg", precision, weak_boundary=True)
    if variant:
        op.set_kernel_variant(variant)
    y, x = product(op, seeded_src(op.m(), 3))
    assert rel_l2(y, weak_oracle(mesh, p).vmult(x)) <= TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n", [(4, 4, 4), (1, 13, 2), (5, 3, 9), (1, 50, 52)])
def test_three_components(cuda, n, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=5)
    op = sf.Operator(mesh, p, "cg", precision, n_components=3)
    op.set_kernel_variant(3)
    y, x = product(op, seeded_src(op.m(), 3))
    o = orc.for_mesh(mesh, p, orc.CG)
    for k in range(3):
        assert rel_l2(y[k::3], o.vmult(np.ascontiguousarray(x[k::3]))) <= TOL[precision]
