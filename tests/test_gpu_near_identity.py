"""Diagonal blocks near the identity, whose factor the Cholesky takes to second order without a first factor
(|S - 1| < 2^-19) or to first order (below 2^-33): matrices on both sides of the two lines, against the
eigenvalues of the oracle's M.

Tolerance: M is good to 1e-13 relative; of the 2 ldim pivots each carries a few roundings of 2^-54 of either
sign, sqrt(300) 2^-54 < 1e-15 for the largest, 5e-15 with a factor of five for their number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ldim", [5, 33, 150])
@pytest.mark.parametrize("bits", [8, 14, 16, 17, 18, 19, 20, 21, 24])
def test_lines(ldim, bits):
    import caps_gb300 as cg
    from oracle import binding as ob
    R, L = 40e-6, 1e-6
    c = cg.Caps(R, L, ldim=ldim, detalg=cg.DETALG_HODLR)
    # log det falls like e^{-2 xi L/c}
    xi = (1 + R / L) / 2 * bits * np.log(2.0)
    got, status = c.logdetD_batch([xi, xi, xi], [0, 1, 4])
    assert (status < 16).all()
    for m, v in zip((0, 1, 4), got):
        want = np.sum(np.log1p(-np.linalg.eigvalsh(ob.M_dense(R, L, ldim, xi, m))))
        assert abs(v - want) <= 1e-12 * abs(want) + 5e-15, (m, v, want)
