"""Learned truncation: samples in batches of 16 per CTA, at the edges of a batch and of the grid."""
import numpy as np
import pytest

import mlp_reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 64, 16 * 304, 16 * 304 + 1, 16 * 608 + 5])
def test_batches(n):
    """FP32 sums of at most 64 terms per neuron and 16 * 3 samples per partial gradient: a few hundred
    roundings of 6e-8 stay below 1e-4 of the largest gradient and 1e-5 of the loss."""
    import caps_gb300 as cg
    net = cg.MLP(seed=7)
    rng = np.random.default_rng(n)
    X = rng.normal(0, 1, (n, 5)).astype(np.float32)
    y = rng.normal(-5, 3, n).astype(np.float32)
    lr, gr, yr = ref.loss_grad(net.params().astype(np.float64), X.astype(np.float64), y.astype(np.float64))
    loss, g = net.loss_grad(X, y)
    assert abs(loss - lr) <= 1e-5 * abs(lr)
    assert np.abs(g - gr).max() <= 1e-4 * np.abs(gr).max()
    assert np.abs(net.predict(X) - yr).max() <= 1e-4 * max(1.0, np.abs(yr).max())
