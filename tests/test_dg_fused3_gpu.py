"""P3 DG / Helmholtz in one launch at the edges of its blocks: fewer cells than a
block, ragged last blocks, cells in random order (nearly every neighbour outside
the block; scalar FP64 then takes two launches); against the oracle."""
import pytest

import oracle as orc
import simplexfem as sf
from test_dg_fused_gpu import KIND, TOL, product, shuffled
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["dg", "helmholtz"])
@pytest.mark.parametrize("mesh", [(1, 1, 1), (3, 7, 1), (8, 8, 2), (9, 5, 7), "shuffled"])
def test_one_launch_matches_oracle(cuda, mesh, kind, precision):
    m = shuffled((6, 5, 7)) if mesh == "shuffled" else sf.Mesh(mesh, jitter=0.1, seed=3)
    op = sf.Operator(m, 3, kind, precision)
    y, x = product(op, seeded_src(op.m(), 2))
    ref = orc.for_mesh(m, 3, KIND[kind], n_components=op.n_components).vmult(x)
    assert rel_l2(y, ref) <= TOL[precision]


@pytest.mark.parametrize("kind", ["dg", "helmholtz"])
def test_one_launch_equals_two(cuda, kind):
    """vmult (one launch) against its two phases (published traces)."""
    import torch
    op = sf.Operator(sf.Mesh((9, 11, 6), jitter=0.1, seed=3), 3, kind)
    x = torch.tensor(seeded_src(op.m(), 2), device="cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)
    op.vmult(a, x)
    op.vmult_phase(b, x, 1)
    op.vmult_phase(b, x, 2)
    assert ((a - b).norm() / b.norm()).item() <= 1e-14
