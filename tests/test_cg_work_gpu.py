"""The bytes that an operator states for a product are those of the tables its form reads."""
import pytest

import simplexfem as sf
from test_cg_patch_gpu import unstructured

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("components", [1, 3])
def test_bytes_by_form(cuda, components):
    """CG P2 FP64 on 24^3 hexes: 216 blocks of 729 nodes (768 codes) and 64 x 36 metric
    values; hexes of 27 DoFs; cells of 10 DoFs and 6 metric values."""
    mesh = sf.Mesh(24, jitter=0.1, seed=1)
    op = sf.Operator(mesh, 2, "cg", n_components=components)
    cells, hexes, vectors = mesh.n_cells, mesh.n_cells // 6, 16 * op.m()
    want = {3: 216 * (4 * 768 + 8 * 36 * 64)}
    if components == 1:
        want.update({2: 48 * cells + 108 * hexes, 5: 48 * cells + 216 * 4 * 729})
        # variant 1 is the patch form here: the metric, then 2 bytes per slot and entry
        # and 4 per distinct DoF of the cells' 10
        op.set_kernel_variant(1)
        assert 48 * cells < op.work()[1] - vectors < (48 + 10 * (2 + 4 + 4)) * cells
    for v, b in want.items():
        op.set_kernel_variant(v)
        assert op.work()[1] == vectors + b, v


def test_bytes_of_a_thread_per_cell(cuda):
    op = sf.Operator(unstructured((4, 4, 4)), 2, "cg")
    assert op.work()[1] == 16 * op.m() + 88 * op.n_cells
