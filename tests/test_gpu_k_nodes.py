"""The quadrature nodes of the K integrals where their rule changes or is stretched: metals whose
Fresnel singularities lie close to the real axis (the bend of the map widens) and far from it,
very low and very high frequencies, the smallest powers at the left end (m = 0, 1) and large m.

The K sums agree with the oracle's adaptive quadrature to about 1e-13; log det is held to the
suite's 1e-10 max(1, |x|), and to 1e-8 relative where it is small."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("metal", [None, (9.0, 0.035), (0.2, 0.05), (0.02, 0.01), (0.001, 0.0005)])
@pytest.mark.parametrize("rl,ldim", [(2.0, 20), (12.0, 40)])
def test_nodes(rl, ldim, metal, mixed):
    import caps_gb300 as cg
    from oracle import binding as ob
    c = cg.Caps(rl * 1e-6, 1e-6, ldim=ldim, detalg=cg.DETALG_LU)
    if metal:
        c.set_drude(*metal)
    if mixed:
        c.set_precision(cg.PREC_MIXED)
    xi = np.array([3e-4, 3e-4, 0.01, 0.1, 1.0, 1.0, 5.0, 20.0])
    m = np.array([0, 1, 2, 1, 0, 7, 3, 1])
    got, status = c.logdetD_batch(xi, m)
    assert (status < 16).all()
    for x, k, v in zip(xi, m, got):
        want = ob.logdetD(rl * 1e-6, 1e-6, ldim, x, k, metal)
        tol, rel = (5e-8, 1e-6) if mixed else (1e-10, 1e-8)
        assert abs(v - want) <= tol * max(1.0, abs(want)) and abs(v - want) <= rel * abs(want) + 1e-12, (x, k, v, want)
