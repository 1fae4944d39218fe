"""Single-pass DG / Helmholtz form (P1, P2) at the edges of its blocks: fewer cells
than a block, ragged last blocks, cells in random order (nearly every neighbour
outside the block), batches of mixed sizes; against the oracle."""
import numpy as np
import pytest

import oracle as orc
import simplexfem as sf
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu

KIND = {"dg": orc.DG, "helmholtz": orc.HELMHOLTZ}
# FP64: the repository's 1e-12; FP32: 2e-6 (tests of the other forms)
TOL = {"fp64": 1e-12, "fp32": 2e-6}


def product(op, x):
    import torch
    src = torch.tensor(x, dtype=op.dtype, device="cuda")
    dst = torch.full_like(src, float("nan"))
    op.vmult(dst, src)
    return dst.double().cpu().numpy(), src.double().cpu().numpy()


def shuffled(n):
    """The box's cells in random order, kept (no reordering)."""
    box = sf.Mesh(n, jitter=0.1, seed=3)
    cells = box.cells()[np.random.default_rng(1).permutation(box.n_cells)]
    return sf.Mesh.from_arrays(box.vertices(), cells, reorder=False)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["dg", "helmholtz"])
@pytest.mark.parametrize("p", [1, 2])
@pytest.mark.parametrize("mesh", [(1, 1, 1), (3, 7, 1), (8, 8, 2), (9, 5, 7), "shuffled"])
def test_single_pass_matches_oracle(cuda, mesh, p, kind, precision):
    m = shuffled((6, 5, 7)) if mesh == "shuffled" else sf.Mesh(mesh, jitter=0.1, seed=3)
    op = sf.Operator(m, p, kind, precision)
    y, x = product(op, seeded_src(op.m(), 2))
    ref = orc.for_mesh(m, p, KIND[kind], n_components=op.n_components).vmult(x)
    assert rel_l2(y, ref) <= TOL[precision]


@pytest.mark.parametrize("p", [1, 2])
def test_single_pass_equals_two_passes(cuda, p):
    """vmult (one pass) against its two phases (published traces)."""
    import torch
    op = sf.Operator(sf.Mesh((9, 11, 6), jitter=0.1, seed=3), p, "dg")
    x = torch.tensor(seeded_src(op.m(), 2), device="cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)
    op.vmult(a, x)
    op.vmult_phase(b, x, 1)
    op.vmult_phase(b, x, 2)
    assert ((a - b).norm() / b.norm()).item() <= 1e-14
