"""Boxes thinner than a block of hexes: the default form of the CG operators is not one
that works for the absent hexes too."""
import pytest

import oracle as orc
import simplexfem as sf
from test_cg_block_gpu import TOL, product
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


def us(op):
    """Best of five times of 20 products."""
    import torch
    x = torch.rand(op.m(), dtype=op.dtype, device="cuda")
    y = torch.empty_like(x)
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = 1e30
    for _ in range(6):
        a.record()
        for _ in range(20):
            op.vmult(y, x)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 50)
    return best


# a quarter (400 x 400 x 1) or half of every block is there: the block form takes two
# to three times as long as the fastest form, so 1.5 tells them apart
@pytest.mark.parametrize("n, p, precision, components, others", [
    ((1, 400, 400), 1, "fp64", 1, (1, 2, 3)), ((1, 400, 400), 2, "fp64", 1, (1, 2, 3)),
    ((1, 400, 400), 2, "fp32", 1, (1, 2, 3)), ((2, 100, 200), 3, "fp32", 3, (1, 3))])
def test_default_is_near_the_fastest_form(cuda, n, p, precision, components, others):
    op = sf.Operator(sf.Mesh(n, jitter=0.1, seed=0), p, "cg", precision, n_components=components)
    default = us(op)
    times = {}
    for v in others:
        op.set_kernel_variant(v)
        times[v] = us(op)
    assert default <= 1.5 * min(times.values()), (default, times)


# forms by the rule's parts: P1 by hexes (50,000 in thin blocks), by patches, by cells
# (few free DoFs), P2 and P3 by patches next to whole and partial blocks
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n, p", [((1, 230, 220), 1), ((5, 5, 120), 1), ((3, 3, 500), 1), ((2, 90, 60), 2),
                                  ((24, 24, 24), 2), ((24, 24, 24), 3), ((21, 22, 23), 3)])
def test_default_form_matches_oracle(cuda, n, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=5)
    op = sf.Operator(mesh, p, "cg", precision)
    y, x = product(op, seeded_src(op.m(), 3))
    assert rel_l2(y, orc.for_mesh(mesh, p, orc.CG).vmult(x)) <= TOL[precision]
