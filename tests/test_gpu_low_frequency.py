"""Extremely low frequencies, where the last quadrature nodes of the K integrals lie at x = nu / (2 xi_), up to 2^205, and
the degree recurrence grows by as much per step.

For perfect reflectors log det(1 - M) tends to the sum of the two xi = 0 blocks (evaluated from closed
forms), from which it differs by terms of the order xi_ or less, below 1e-8 here.  Bar: the suite's 1e-10
max(1, |x|), and 1e-8 relative where it is small (the xi = 0 blocks take the trace rule below 1e-8 each, good
to half that)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

XI = np.array([1e-8, 1e-10, 1e-11, 1e-12, 1e-13, 1e-14, 1e-15, 1e-16, 1e-17, 1e-18, 1e-20, 1e-25, 1e-40, 1e-60])


@pytest.mark.parametrize("m", [0, 1, 2, 30, 100])
@pytest.mark.parametrize("rl,ldim", [(20.0, 140), (150.0, 300)])
def test_limit(rl, ldim, m):
    import caps_gb300 as cg
    c = cg.Caps(rl * 1e-6, 1e-6, ldim=ldim, detalg=cg.DETALG_LU)
    want = sum(c.logdetD0(m))
    got, status = c.logdetD_batch(XI, np.full(len(XI), m))
    assert (status < 16).all()
    for x, v in zip(XI, got):
        assert abs(v - want) <= 1e-10 * max(1.0, abs(want)) and abs(v - want) <= 1e-8 * abs(want), (x, m, v, want)


@pytest.mark.parametrize("rl,m", [(300.0, 1500), (1000.0, 400)])
@pytest.mark.parametrize("xi", [1e-9, 1e-11, 1e-12, 1e-14, 1e-15])
def test_large_m(rl, m, xi):
    """large m, where the recurrence's first coefficient 2 mu + 1 counts too: against a frequency so much higher that
    its nodes stay below 2^32, but low enough to share the limit (terms of the order xi_^2)"""
    import caps_gb300 as cg
    c = cg.Caps(rl * 1e-6, 1e-6, ldim=200, detalg=cg.DETALG_LU)
    (got, want), status = c.logdetD_batch([xi, 1e-5], [m, m])
    assert (status < 16).all()
    assert want != 0 and abs(got - want) <= 1e-8 * abs(want), (got, want)
