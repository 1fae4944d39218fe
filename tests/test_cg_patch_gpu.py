"""CG operators by patches of cells: unstructured meshes around the smallest size
that goes by patches, a last patch of one cell, cells in an order without
neighbours (FP64 and P2: thread per cell), boxes without blocks enough, three components;
against the oracle."""
import numpy as np
import pytest

import oracle as orc
import simplexfem as sf
from test_cg_block_gpu import TOL, product
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


def unstructured(n, cells=None, reorder=True):
    """A box's first `cells` cells with shuffled numbering, ordered by the library or not."""
    box = sf.Mesh(n, jitter=0.1, seed=3)
    rng = np.random.default_rng(2)
    new = rng.permutation(box.n_vertices)
    vertices = np.empty_like(box.vertices())
    vertices[new] = box.vertices()
    c = new[box.cells()[:cells]]
    used = np.unique(c)
    c = np.searchsorted(used, c)
    return sf.Mesh.from_arrays(vertices[used], c[rng.permutation(len(c))], reorder=reorder)


MESHES = {
    "191 patches": lambda: unstructured((16, 16, 16), 191 * 128),
    "192 patches, 1 cell": lambda: unstructured((16, 16, 16), 191 * 128 + 1),
    "255 patches": lambda: unstructured((18, 18, 18), 255 * 128),
    "256 patches, 1 cell": lambda: unstructured((18, 18, 18), 255 * 128 + 1),
    "274 patches": lambda: unstructured((18, 18, 18)),
    "random order": lambda: unstructured((18, 18, 18), reorder=False),
    "few blocks": lambda: sf.Mesh((8, 27, 27), jitter=0.1, seed=3),
}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("mesh", MESHES)
def test_patches_match_oracle(cuda, mesh, p, precision):
    m = MESHES[mesh]()
    op = sf.Operator(m, p, "cg", precision)
    y, x = product(op, seeded_src(op.m(), 3))
    assert rel_l2(y, orc.for_mesh(m, p, orc.CG).vmult(x)) <= TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n, cells", [((14, 14, 14), None), ((13, 13, 13), 191 * 64 + 33)])
def test_three_components_by_patches(cuda, n, cells, p, precision):
    m = unstructured(n, cells)
    op = sf.Operator(m, p, "cg", precision, n_components=3)
    y, x = product(op, seeded_src(op.m(), 3))
    o = orc.for_mesh(m, p, orc.CG)
    for k in range(3):
        assert rel_l2(y[k::3], o.vmult(np.ascontiguousarray(x[k::3]))) <= TOL[precision]
