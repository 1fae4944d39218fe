"""Block and patch forms of the CG operator on the parts of a partitioned box:
partly filled blocks at the cut, DoFs that are interior to a block or a patch only
among the part's own cells, identity rows of owned DoFs only; against the oracle
(small boxes) and the whole operator with a thread per cell."""
import pytest

import oracle as orc
import simplexfem as sf
from test_cg_block_gpu import TOL, product
from test_partition_gpu import partitioned_vmult
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


def free_src(mesh, p, precision):
    op = sf.Operator(mesh, p, "cg", precision)
    return op, seeded_src(op.m(), 3, op.constrained())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n, parts", [((9, 10, 7), 3), ((5, 3, 9), 2), ((4, 4, 4), 4)])
def test_block_form_on_parts(cuda, n, parts, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=1)
    _, x = free_src(mesh, p, precision)
    y = partitioned_vmult(mesh, p, "cg", 1, parts, x, precision=precision, variant=3)
    assert rel_l2(y, orc.for_mesh(mesh, p, orc.CG).vmult(x)) <= TOL[precision]


# 24 x 24 x 48: about 216 blocks a part, several resident ones an SM; 18 x 18 x 36: about
# 273 patches a part, patches by default
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n, variant", [((24, 24, 48), 3), ((18, 18, 36), 0)])
def test_larger_parts(cuda, n, variant, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=1)
    op, x = free_src(mesh, p, precision)
    y = partitioned_vmult(mesh, p, "cg", 1, 2, x, precision=precision, variant=variant)
    op.set_kernel_variant(1)
    assert rel_l2(y, product(op, x)[0]) <= TOL[precision]
