"""The recurrence's rows in parts, each but the first from the q-sums of two whole rows: from ldim 1024 on in both forms, one
more part at 1536, the number by ldim alone.

FP64 against HODLR, which forms every element it needs by q-sums, at the suite's 1e-10 max(1, |x|); the mixed form
against FP64 at its 5e-8.  A matrix has the same bits alone and in a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
METALS = [None, (9.0, 0.035)]


@pytest.mark.parametrize("ldim", [1023, 1024, 1535, 1536])
@pytest.mark.parametrize("metal", METALS)
def test_lines(ldim, metal):
    import caps_gb300 as cg
    c = cg.Caps(180e-6, 1e-6, ldim=ldim)
    if metal:
        c.set_drude(*metal)
    xi, m = np.array([2.0, 40.0, 40.0, 90.0, 250.0]), np.array([0, 1, 30, 0, 3])
    got = {}
    for name, path, prec in (("hodlr", cg.PATH_HODLR, cg.PREC_FP64), ("dense", cg.PATH_DENSE, cg.PREC_FP64),
                             ("mixed", cg.PATH_DENSE, cg.PREC_MIXED)):
        c.set_path(path)
        c.set_precision(prec)
        got[name], status = c.logdetD_batch(xi, m)
        assert (status == 3).all(), (name, status)
    scale = np.maximum(1.0, np.abs(got["hodlr"]))
    assert (np.abs(got["dense"] - got["hodlr"]) <= 1e-10 * scale).all(), got
    assert (np.abs(got["mixed"] - got["dense"]) <= 5e-8 * scale).all(), got


@pytest.mark.parametrize("ldim", [1024, 1536])
@pytest.mark.parametrize("mixed", [False, True])
def test_alone_and_in_a_batch(ldim, mixed):
    import caps_gb300 as cg
    c = cg.Caps(180e-6, 1e-6, ldim=ldim)
    c.set_drude(9.0, 0.035)
    c.set_path(cg.PATH_DENSE)
    if mixed:
        c.set_precision(cg.PREC_MIXED)
    xi, m = np.tile([30.0, 200.0], 10), np.repeat(np.arange(10), 2)
    many, status = c.logdetD_batch(xi, m)
    assert (status < 16).all()
    for k in (0, 1, 7, 19):
        assert c.logdetD(xi[k], m[k]) == many[k]
