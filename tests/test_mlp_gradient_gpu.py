"""Training gradient at the edges of its tiles and grids, against the FP64 oracle."""
import numpy as np
import pytest

import mlp_oracle
import simplexfem as sf

pytestmark = pytest.mark.gpu


# 16-sample tiles up to one per SM (148 x 16 = 2368), 32-sample tiles above,
# several tiles per CTA above 2 x 148 x 32 = 9472
@pytest.mark.parametrize("n", [1, 15, 16, 17, 2368, 2369, 9473])
def test_gradient_at_tile_edges(cuda, n):
    import torch
    mlp = sf.MLP(seed=3)
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 29)).astype(np.float32)
    Y = rng.standard_normal((n, 20)).astype(np.float32)
    g, loss = mlp.gradient(torch.tensor(X, device="cuda"), torch.tensor(Y, device="cuda"))
    ref_loss, ref_g = mlp_oracle.loss_and_grad(mlp.weights(), X, Y)
    # FP32 sums of at most a few hundred terms per stage (64 inputs, 32 samples,
    # 296 CTAs): 2^-24 times that is below 2e-5
    assert abs(loss - ref_loss) <= 2e-5 * ref_loss
    assert np.linalg.norm(g.cpu().numpy() - ref_g) <= 2e-5 * np.linalg.norm(ref_g)
