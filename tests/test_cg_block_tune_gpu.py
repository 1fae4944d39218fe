"""The autotuner also times the block form of CG where that is the default."""
import pytest

import oracle as orc
import simplexfem as sf
from test_cg_block_gpu import TOL, product
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("components", [1, 3])
def test_autotuner_times_the_block_form(cuda, components):
    sf.set_autotune_cache(None)
    mesh = sf.Mesh((24, 24, 24), jitter=0.1, seed=5)
    op = sf.Operator(mesh, 2, "cg", "fp64", n_components=components)
    r = op.autotune(reps=3, use_cache=False)
    assert r["us"][2] > 0
    y, x = product(op, seeded_src(op.m(), 2))
    o = orc.for_mesh(mesh, 2, orc.CG)
    for k in range(components):
        assert rel_l2(y[k::components], o.vmult(x[k::components].copy())) <= TOL["fp64"]
