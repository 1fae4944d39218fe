"""p-transfers by blocks on a box whose last blocks are padded (22 hexes: five blocks
of four and one of two), with strong and with weak boundary conditions (no constrained
nodes), against the embedding matrix applied cell by cell."""
import numpy as np
import pytest

import simplexfem as sf
from test_mg_block_transfer_gpu import TOL, reference

pytestmark = pytest.mark.gpu


class Unconstrained:
    def __init__(self, mesh):
        self.mesh = mesh

    def cg_dofs(self, p):
        dofs, fixed = self.mesh.cg_dofs(p)
        return dofs, np.zeros_like(fixed)


@pytest.mark.parametrize("precision, weak", [("fp64", False), ("fp32", False), ("fp32", True)])
def test_p_transfers_of_padded_blocks(cuda, precision, weak):
    import torch
    mesh = sf.Mesh(22, jitter=0.05, seed=1)
    op = sf.Operator(mesh, 3, "dg" if weak else "cg")
    mg = sf.Multigrid(op, precision=precision, coarse_n=11, c_transfer=int(weak), weak_cg_levels=weak)
    dt = torch.float64 if precision == "fp64" else torch.float32
    rng = np.random.default_rng(3)
    for p in (2, 3):  # levels: P1 on 11^3, then P1, P2, P3 on 22^3
        assert mg.level_info(p)["degree"] == p and mg.level_info(p)["kind"] == "cg"
        xc, xf = (rng.uniform(-1, 1, mg.level_info(k)["m"]) for k in (p - 1, p))
        c, f = torch.tensor(xc, dtype=dt, device="cuda"), torch.tensor(xf, dtype=dt, device="cuda")
        fine, coarse = reference(Unconstrained(mesh) if weak else mesh, p, c.double().cpu().numpy(),
                                 f.double().cpu().numpy())
        out = torch.ones_like(f)
        mg.prolongate_add(p, out, c)
        # rounding of 1 + x, as at the unpadded sizes
        assert np.linalg.norm(out.double().cpu().numpy() - 1.0 - fine) <= 4 * TOL[precision] * np.sqrt(len(fine))
        out = torch.zeros_like(c)
        mg.restrict_add(p, out, f)
        assert np.linalg.norm(out.double().cpu().numpy() - coarse) <= TOL[precision] * np.linalg.norm(coarse)
