"""Learned truncation: the networks of a process share one block of pinned memory that samples and results pass through.
Sizes on both sides of what fits (16384 samples with their values, 19660 without, 98304 predictions), and networks
of several threads at once: the values of a network used alone."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def data(n, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (n, 5)).astype(np.float32), rng.normal(-5, 3, n).astype(np.float32)


@pytest.mark.parametrize("n", [16384, 16385, 19660, 19661, 98304, 98305])
def test_sizes(n):
    """predictions are those of the samples' parts; loss and gradient are their weighted means, FP32 sums of a few hundred
    thousand terms in another order"""
    import caps_gb300 as cg
    net = cg.MLP(seed=11)
    X, y = data(n, n)
    h = n // 2
    got = net.predict(X)
    assert (got == np.concatenate([net.predict(X[:h]), net.predict(X[h:])])).all()
    loss, g = net.loss_grad(X, y)
    (l1, g1), (l2, g2) = net.loss_grad(X[:h], y[:h]), net.loss_grad(X[h:], y[h:])
    assert abs(loss - (h * l1 + (n - h) * l2) / n) <= 1e-5 * abs(loss)
    assert np.abs(g - (h * g1 + (n - h) * g2) / n).max() <= 1e-4 * np.abs(g).max()


def test_threads():
    import caps_gb300 as cg

    def work(k):
        out = []
        for i in range(12):
            net = cg.MLP(seed=100 * k + i)
            X, y = data(50 + 700 * k + i, 1000 * k + i)
            loss = net.train(X, y, epochs=3)
            out.append((loss, *net.loss_grad(X, y), net.predict(X)))
            del net
        return out
    alone = [work(k) for k in range(4)]
    with ThreadPoolExecutor(4) as ex:
        together = list(ex.map(work, range(4)))
    for a, b in zip(alone, together):
        for u, v in zip(a, b):
            assert u[0] == v[0] and u[1] == v[1] and (u[2] == v[2]).all() and (u[3] == v[3]).all()
