"""The estimator's tiled gradient kernel at the edges of its tiles and of its grid (GPU).

k_mlp_grad works on tiles of 32 samples with at most 296 CTAs: one sample, a
full tile and its neighbours, the largest single pass (9472 samples) and one
more, and a size where some CTAs take several tiles.  Tolerance: FP32 dot
products of up to 64 terms per layer and sums over the samples with random
rounding, as in the gradient test of test_gpu_mlp.py.
"""
import numpy as np
import pytest

import sjoin
from oracle import mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 32, 33, 9472, 9473, 20011])
def test_gradient_at_tile_edges(m):
    rng = np.random.default_rng(m)
    x = rng.standard_normal((m, 16)).astype(np.float32)
    t = np.stack([x[:, :4].sum(1), np.abs(x[:, 4:8]).sum(1)], 1).astype(np.float32)
    w = sjoin.mlp_init(5)
    loss, g = sjoin.mlp_loss_grad(x, t, w)
    rloss, rg = mlp.loss_grad(x, t, w.astype(np.float64))
    assert abs(loss - rloss) <= 1e-4 * max(1.0, abs(rloss))
    np.testing.assert_allclose(g, rg, rtol=2e-3, atol=2e-5 * max(1.0, np.abs(rg).max()))
    again = sjoin.mlp_loss_grad(x, t, w)
    assert again[0] == loss and np.array_equal(again[1], g)   # fixed order of the sums
