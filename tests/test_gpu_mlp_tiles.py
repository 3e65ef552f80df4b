"""The network's tiled kernels at the sizes where their tiling changes: one sample, the edges of
a 16-sample tile, and more tiles than resident CTAs (each CTA then walks several tiles)."""
import numpy as np
import pytest

from oracle import selector_ref as R
from pava_b200 import selector as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 15, 16, 17, 33, 4800, 9500])
def test_forward_and_gradient_across_tiles(cuda, B):
    rng = np.random.default_rng(B)
    X = rng.normal(size=(B, R.IN)).astype(np.float32)
    T = rng.normal(size=(B, R.OUT)).astype(np.float32)
    mask = (rng.uniform(size=(B, R.OUT)) > 0.1).astype(np.float32)
    net = S.Network(seed=B + 1)
    P, _, _ = net.params()
    # FP32 chains of at most 64 terms of magnitude O(1): 64 * 2^-24 * a few
    Yr, _ = R.mlp_forward(P, X.astype(np.float64))
    assert np.max(np.abs(net.forward(X) - Yr)) <= 64 * 2.0 ** -24 * 8 * max(1.0, np.abs(Yr).max())
    net.set_batch(X, T, mask)
    loss, g = net.gradient()
    lr, gr = R.mlp_loss_grad(P, X, T, mask)
    assert abs(loss - lr) <= 1e-5 * max(1.0, abs(lr))
    # the bound of the untiled gradient test: 1e-4 of the largest entry
    assert np.max(np.abs(g - gr)) <= 1e-4 * np.abs(gr).max()
    assert np.array_equal(g, net.gradient()[1])  # fixed order: same bits
