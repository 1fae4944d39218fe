"""Tables of the DG and Helmholtz kernel forms: an operator in one launch holds its blocked
geometry only; geometry by cells and the trace buffer are made when a two-launch form,
a phase or the diagonal is asked for."""
import pytest

import oracle as orc
import simplexfem as sf
from test_cg_tables_gpu import used
from test_dg_fused_gpu import KIND, TOL, product, shuffled
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


# bytes per cell in FP64: 22 (P3: 10) values, with mass one more, face codes (8, P3 16),
# 4 per outer neighbour and 36 (P3) per outer face, at most one of each per cell
@pytest.mark.parametrize("p, kind, size", [(1, "dg", 188), (2, "dg", 188), (3, "dg", 136), (2, "helmholtz", 196),
                                           (3, "helmholtz", 144)])
def test_memory_of_the_default_form(cuda, p, kind, size):
    mesh = sf.Mesh(48, jitter=0.1, seed=1)
    sf.Operator(mesh, p, kind)  # modules and heaps are loaded
    before = used()
    op = sf.Operator(mesh, p, kind)
    assert used() - before <= size * mesh.n_cells + (16 << 20)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["dg", "helmholtz"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("mesh", [(9, 5, 7), "shuffled"])
def test_made_on_demand(cuda, mesh, p, kind, precision):
    import torch
    m = shuffled((6, 5, 7)) if mesh == "shuffled" else sf.Mesh(mesh, jitter=0.1, seed=3)
    op = sf.Operator(m, p, kind, precision)
    ref = orc.for_mesh(m, p, KIND[kind], n_components=op.n_components)
    d = op.initialize_dof_vector()
    op.compute_diagonal(d)
    assert rel_l2(d.double().cpu().numpy(), ref.diagonal()) <= TOL[precision]
    x = torch.tensor(seeded_src(op.m(), 2), dtype=op.dtype, device="cuda")
    want = ref.vmult(x.double().cpu().numpy())
    y = torch.full_like(x, float("nan"))
    op.vmult_phase(y, x, 1)
    op.vmult_phase(y, x, 2)
    assert rel_l2(y.double().cpu().numpy(), want) <= TOL[precision]
    op = sf.Operator(m, p, kind, precision)
    for v in (3, 1, 2, 5, 0):
        op.set_kernel_variant(v)
        assert rel_l2(product(op, seeded_src(op.m(), 2))[0], want) <= TOL[precision], v


def test_phases_while_capturing(cuda):
    import torch
    op = sf.Operator(sf.Mesh((9, 5, 7), jitter=0.1, seed=3), 2, "dg")
    x = torch.tensor(seeded_src(op.m(), 2), device="cuda")
    want, got, diag = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    op.vmult(want, x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        op.vmult_phase(got, x, 1)
        op.vmult_phase(got, x, 2)
        op.compute_diagonal(diag)
    g.replay()
    d = torch.empty_like(x)
    op.compute_diagonal(d)
    torch.cuda.synchronize()
    assert rel_l2(got.cpu().numpy(), want.cpu().numpy()) <= 1e-14
    assert torch.equal(d, diag)


@pytest.mark.parametrize("variant", [1, 2, 3])
def test_batch_forms(cuda, variant):
    import torch
    ops = [sf.Operator(sf.Mesh(n, jitter=0.1, seed=3), 3, "helmholtz") for n in ((1, 1, 1), (4, 3, 5))]
    xs = [torch.tensor(seeded_src(o.m(), 5), device="cuda") for o in ops]
    ys = [torch.full_like(x, float("nan")) for x in xs]
    b = sf.Batch(ops)
    b.set_kernel_variant(variant)
    b.vmult(ys, xs)
    for o, x, y in zip(ops, xs, ys):
        ref = orc.for_mesh(o.mesh, 3, orc.HELMHOLTZ, n_components=3).vmult(x.cpu().numpy())
        assert rel_l2(y.cpu().numpy(), ref) <= 1e-12
