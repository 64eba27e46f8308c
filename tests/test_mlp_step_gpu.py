"""The training step's kernel at partial chunks (128 samples, 32 per CTA) and many of them:
gradients against the FP64 restatement, with the bounds of test_mlp_gpu.py."""
import numpy as np
import pytest

import mlp_oracle as M
import psift

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 97, 127, 128, 129, 300, 20001])
def test_gradients_at_partial_chunks(n):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 8)).astype(np.float32)
    Y = (rng.random(n) < 0.5).astype(np.float32)
    mlp = psift.InlierMLP(seed=6)
    loss, g = mlp.gradients(X, Y)
    rloss, rg = M.loss_and_grad(mlp.params, X, Y)
    assert abs(loss - rloss) < 1e-4 * max(1.0, abs(rloss))
    assert np.linalg.norm(g - rg) <= 2e-3 * np.linalg.norm(rg)
