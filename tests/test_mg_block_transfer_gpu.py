"""p-transfers by blocks of hexes against the embedding matrix applied cell by cell
(numpy), at box sizes of one wave of blocks and of more."""
import numpy as np
import pytest

import gen_tables
import simplexfem as sf

pytestmark = pytest.mark.gpu
EMB = {p: np.array([[float(v) for v in r] for r in gen_tables.build()[p]["EMB"]]) for p in (2, 3)}
# interpolation with at most 6 terms of weight below 1, restriction sums of at most
# about 60 x 24 terms: a few ten roundings
TOL = {"fp64": 1e-14, "fp32": 1e-6}


def reference(mesh, p, xc, xf):
    """(P xc added to zero, P^T xf) over the free nodes."""
    df, mf = mesh.cg_dofs(p)
    dc, mc = mesh.cg_dofs(p - 1)
    uc = np.where(mc.astype(bool), 0.0, xc)
    fine = np.zeros(len(mf))
    fine[df] = uc[dc] @ EMB[p].T
    fine[mf.astype(bool)] = 0.0
    first = np.full(len(mf), -1)
    flat = df.reshape(-1)
    first[flat[::-1]] = np.arange(flat.size)[::-1]  # the first cell-local place of every fine node
    r = np.where(mf.astype(bool), 0.0, xf)
    coarse = np.zeros(len(mc))
    cell, loc = first // df.shape[1], first % df.shape[1]
    np.add.at(coarse, dc[cell], EMB[p][loc] * r[:, None])
    coarse[mc.astype(bool)] = 0.0
    return fine, coarse


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n, p", [(24, 2), (24, 3), (32, 2), (32, 3)])
def test_p_transfers(cuda, n, p, precision):
    import torch
    mesh = sf.Mesh(n, jitter=0.05, seed=1)
    op = sf.Operator(mesh, p, "cg")
    mg = sf.Multigrid(op, precision=precision, coarse_n=3 if n == 24 else 4)
    top = mg.n_levels - 1
    dt = torch.float64 if precision == "fp64" else torch.float32
    rng = np.random.default_rng(3)
    xc, xf = rng.uniform(-1, 1, mg.level_info(top - 1)["m"]), rng.uniform(-1, 1, op.m())
    c, f = torch.tensor(xc, dtype=dt, device="cuda"), torch.tensor(xf, dtype=dt, device="cuda")
    fine, coarse = reference(mesh, p, c.double().cpu().numpy(), f.double().cpu().numpy())
    out = torch.ones_like(f)
    mg.prolongate_add(top, out, c)
    got = out.double().cpu().numpy() - 1.0
    assert np.linalg.norm(got - fine) <= 4 * TOL[precision] * np.sqrt(len(fine))  # rounding of 1 + x
    out = torch.zeros_like(c)
    mg.restrict_add(top, out, f)
    assert np.linalg.norm(out.double().cpu().numpy() - coarse) <= TOL[precision] * np.linalg.norm(coarse)
