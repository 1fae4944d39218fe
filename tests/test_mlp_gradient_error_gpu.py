"""Error of the training gradient against 64 bits: no larger than that of a sum of
few partial sums, whatever the number of CTAs."""
import numpy as np
import pytest

import mlp_oracle
import simplexfem as sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700, 2048, 8192])
def test_gradient_error(cuda, n):
    """G partial sums added one after another onto a growing total round G times, the
    k-th time at k / G of the result: sqrt(G / 3) roundings of rms 0.42 2^-24 (the
    mean over the mantissa of a relative rounding of at most 2^-24, uniform).  The
    128-sample partial sums of one CTA each are G = n / 128; the rest of the error
    (activations, sums inside a partial sum), independent of it, gets as much again,
    and no less than one and a half roundings in all."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    r = torch.randn(n, 20, generator=g, device="cuda")
    r /= r.norm(dim=1, keepdim=True)
    j = torch.eye(3, device="cuda").reshape(1, 9) + 0.3 * torch.randn(n, 9, generator=g, device="cuda")
    Y = 0.3 * r + 0.1 * torch.randn(n, 20, generator=g, device="cuda")
    X = torch.cat([r, j], 1).contiguous()
    mlp = sf.MLP(seed=1)
    got, _ = mlp.gradient(X, Y)
    _, ref = mlp_oracle.loss_and_grad(mlp.weights(), X.cpu().numpy(), Y.cpu().numpy())
    tol = max(np.sqrt(2) * 0.42 * np.sqrt(n / 128 / 3), 1.5) * 2.0 ** -24
    assert np.linalg.norm(got.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
