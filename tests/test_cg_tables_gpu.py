"""Tables of the CG kernel forms: an operator holds those of the form it runs, others are
made when they are asked for."""
import pytest

import oracle as orc
import simplexfem as sf
from test_cg_block_gpu import TOL, product
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


def used():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_memory_of_the_default_form(cuda):
    """CG P2 FP64, bytes per cell: 40 DoF table, 48 metric, 48 metric by blocks, 8 and 8
    block and cube codes; the hex form's 48 + 18 come with variant 2."""
    mesh = sf.Mesh(64, jitter=0.1, seed=1)
    sf.Operator(mesh, 2, "cg")  # modules and heaps are loaded
    before = used()
    op = sf.Operator(mesh, 2, "cg")
    made = used()
    assert made - before <= 152 * mesh.n_cells + (16 << 20)
    op.set_kernel_variant(2)
    hexes = used()
    assert 0.9 * 66 * mesh.n_cells <= hexes - made <= 66 * mesh.n_cells + (16 << 20)
    for v in (1, 2, 3, 5, 0):
        op.set_kernel_variant(v)
    assert used() <= hexes + (16 << 20)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n", [(5, 3, 9), (8, 8, 4), (1, 13, 2)])
def test_forms_in_any_order(cuda, n, p, precision):
    mesh = sf.Mesh(n, jitter=0.1, seed=5)
    ref = orc.for_mesh(mesh, p, orc.CG)
    for order in ((3, 2, 1), (5, 3), (2, 0, 3, 7)):
        op = sf.Operator(mesh, p, "cg", precision)
        for v in order:
            op.set_kernel_variant(v)
            y, x = product(op, seeded_src(op.m(), 3))
            assert rel_l2(y, ref.vmult(x)) <= TOL[precision], v


@pytest.mark.parametrize("components", [1, 3])
def test_forms_switched_while_capturing(cuda, components):
    import torch
    mesh = sf.Mesh((9, 8, 7), jitter=0.1, seed=5)
    op = sf.Operator(mesh, 2, "cg", n_components=components)
    x = torch.tensor(seeded_src(op.m(), 3), device="cuda")
    want = torch.empty_like(x)
    op.vmult(want, x)
    out = [torch.full_like(x, float("nan")) for _ in range(3)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for y, v in zip(out, (2, 3, 1)):
            op.set_kernel_variant(v)
            op.vmult(y, x)
    g.replay()
    torch.cuda.synchronize()
    for y in out:
        assert rel_l2(y.cpu().numpy(), want.cpu().numpy()) <= TOL["fp64"]
