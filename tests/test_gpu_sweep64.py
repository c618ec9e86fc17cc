"""The FP64 form's recurrence (dense path) where it can go wrong: the smallest windows, both
sides of the 30-column passes, rows split over several CTAs or not (few or many matrices of one
batch), windows that start above m, the ring of rows in shared and in global memory.

Bar: the suite's 1e-10 max(1, |x|) against the oracle, which sums every pair; seeds of the
recurrence carry that algorithm's rounding (about 1e-13), and it moves away from them by
coefficients of order one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
METALS = [None, (9.0, 0.035), (9.0, 0.0)]


@pytest.mark.parametrize("ldim", [1, 2, 3, 4, 5, 29, 30, 31, 59, 60, 61, 127, 128, 129, 200])
@pytest.mark.parametrize("metal", METALS)
def test_windows(ldim, metal):
    import caps_gb300 as cg
    from oracle import binding as ob
    R, L = 25e-6, 1e-6
    c = cg.Caps(R, L, ldim=ldim, detalg=cg.DETALG_LU)
    if metal:
        c.set_drude(*metal)
    xi, m = np.array([0.3, 6.0, 40.0, 3.0]), np.array([0, 1, 2, 30])
    got, status = c.logdetD_batch(xi, m)
    assert (status < 16).all()
    for k in range(4):
        want = ob.logdetD(R, L, ldim, xi[k], m[k], metal)
        assert abs(got[k] - want) <= 1e-10 * max(1.0, abs(want)), (ldim, metal, xi[k], m[k], got[k], want)


@pytest.mark.parametrize("ldim", [128, 300, 520])
def test_row_parts(ldim):
    """a batch of one matrix splits its rows, a batch of 200 does not: the same values"""
    import caps_gb300 as cg
    c = cg.Caps(70e-6, 1e-6, ldim=ldim)
    c.set_drude(9.0, 0.035)
    xi, m = np.tile([9.0, 60.0], 100), np.repeat(np.arange(20), 10)
    many, status = c.logdetD_batch(xi, m)
    assert (status < 16).all()
    for k in (0, 1, 57, 130):
        one = c.logdetD(xi[k], m[k])
        assert abs(one - many[k]) <= 1e-12 * max(1.0, abs(one)), (k, one, many[k])


def test_ring_in_global_memory():
    """a window beyond the shared-memory ring against HODLR, which forms its elements by q-sums"""
    import caps_gb300 as cg
    c = cg.Caps(500e-6, 1e-6, ldim=3600)
    c.set_drude(9.0, 0.0)
    c.set_path(cg.PATH_DENSE)
    dense = c.logdetD(300.0, 1)
    c.set_path(cg.PATH_HODLR)
    hodlr = c.logdetD(300.0, 1)
    assert abs(dense - hodlr) <= 1e-10 * max(1.0, abs(hodlr)), (dense, hodlr)


@pytest.mark.parametrize("ldim", [16, 17, 64, 65, 130, 260])
@pytest.mark.parametrize("metal", METALS)
def test_elements_that_round_to_zero(ldim, metal):
    """HODLR rules skip elements that round to zero, the dense rules (which need |M|) form every one: the
    same fixed-point matrix, so the same bits wherever both factor it"""
    import caps_gb300 as cg
    xi = np.array([0.2, 2.0, 9.0, 25.0]) * 10
    m = np.array([1, 0, 4, 2])
    out = []
    for alg in (cg.DETALG_LU, cg.DETALG_HODLR):
        c = cg.Caps(40e-6, 1e-6, ldim=ldim, detalg=alg)
        if metal:
            c.set_drude(*metal)
        out.append(c.logdetD_batch(xi, m))
    both = (out[0][1] == 3) & (out[1][1] == 3)
    assert both.sum() >= 2
    assert (out[0][0][both] == out[1][0][both]).all()


def test_ring_beyond_shared_memory():
    """one row of one polarisation no longer fits shared memory four times: against HODLR as above"""
    import caps_gb300 as cg
    c = cg.Caps(900e-6, 1e-6, ldim=7100)
    c.set_drude(9.0, 0.0)
    c.set_path(cg.PATH_DENSE)
    dense = c.logdetD(900.0, 1)
    c.set_path(cg.PATH_HODLR)
    hodlr = c.logdetD(900.0, 1)
    assert abs(dense - hodlr) <= 1e-10 * max(1.0, abs(hodlr)), (dense, hodlr)
