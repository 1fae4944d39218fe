"""Batched Helmholtz launches of every degree: problems of mixed sizes, fewer cells
than a block among them, one with its cells in random order (which sets the shared
memory of the whole launch and, for scalar P3 FP64, sends it to two launches), one
operator listed twice; against single products and the oracle."""
import pytest

import oracle as orc
import simplexfem as sf
from test_dg_fused_gpu import TOL, shuffled
from util import rel_l2, seeded_src

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["dg", "helmholtz"])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_batch_equals_single_products(cuda, p, kind, precision, mixed):
    import torch
    meshes = [sf.Mesh(n, jitter=0.1, seed=3) for n in ((1, 1, 1), (9, 5, 7), (4, 3, 5))]
    if mixed:
        meshes.append(shuffled((6, 5, 7)))
    ops = [sf.Operator(m, p, kind, precision) for m in meshes]
    ops.append(ops[1])
    xs = [torch.tensor(seeded_src(o.m(), 5 + k), dtype=o.dtype, device="cuda") for k, o in enumerate(ops)]
    ys = [torch.full_like(x, float("nan")) for x in xs]
    sf.Batch(ops).vmult(ys, xs)
    okind = {"dg": orc.DG, "helmholtz": orc.HELMHOLTZ}[kind]
    for o, x, y in zip(ops, xs, ys):
        one = torch.empty_like(x)
        o.vmult(one, x)
        # the same kernel, or (one problem's order) its two-launch form: rounding
        assert rel_l2(y.double().cpu().numpy(), one.double().cpu().numpy()) <= TOL[precision]
        ref = orc.for_mesh(o.mesh, p, okind, n_components=o.n_components).vmult(x.double().cpu().numpy())
        assert rel_l2(y.double().cpu().numpy(), ref) <= TOL[precision]
