"""Cylinder-plane: the Bessel tables over their range (small and large arguments, Hankel's expansion of I_0 above
2000, orders that need rescaling) and elements at the edges of the 64 x 16 blocks.

Reference: the oracle's FP64 restatement.  Tolerance: as for the factorisation, 1e-12 max(1, |x|) + 1e-14 n; where
the trace rule decides (|x| < 1e-8) the value is a sum of positive products of three table entries, each of a
chain of at most 900 roundings of 2^-53 of either sign, and the oracle's of exponentials of logarithms of
magnitude up to 10^3: 1e-9 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 16, 17, 64, 65, 150])
@pytest.mark.parametrize("boundary", ["D", "N"])
@pytest.mark.parametrize("ratio", [0.5, 20.0, 150.0])
def test_arguments(n, boundary, ratio):
    import caps_gb300 as cg
    from oracle import binding as ob
    d = 1e-6
    R = ratio * d
    q = np.array([1e-5, 1e-2, 0.3, 2.0, 9.0, 30.0]) / (2 * d)
    got = cg.capc_logdet(R, d, q, boundary, n, "LU")
    for x, v in zip(q, got):
        want = ob.lib.oracle_capc_logdet(R, d, n, float(x), boundary.encode(), 0)
        tol = 1e-9 * abs(want) if abs(want) < 1e-8 else 1e-12 * max(1.0, abs(want)) + 1e-14 * n
        assert abs(v - want) <= tol, (x, v, want)
