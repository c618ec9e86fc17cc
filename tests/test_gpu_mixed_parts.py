"""Mixed form, windows whose rows are split into parts that start from two rows of q-sums: both sides of the line
(ldim 2230) and of a change of their number, against the FP64 form.  Bar: the mixed form's 5e-8 max(1, |x|)
of the suite; the recurrence itself moves log det by 5e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ldim", [2229, 2230, 2231, 2559, 2560])
@pytest.mark.parametrize("metal", [None, (9.0, 0.035)])
def test_parts(ldim, metal):
    import caps_gb300 as cg
    xi, m = np.array([3.0, 40.0, 250.0]), np.array([0, 1, 9])
    out = []
    for prec in (cg.PREC_FP64, cg.PREC_MIXED):
        c = cg.Caps(320e-6, 1e-6, ldim=ldim)
        if metal:
            c.set_drude(*metal)
        c.set_path(cg.PATH_DENSE)
        c.set_precision(prec)
        out.append(c.logdetD_batch(xi, m))
    assert (out[0][1] < 16).all() and (out[1][1] < 16).all()
    assert (np.abs(out[0][0] - out[1][0]) <= 5e-8 * np.maximum(1.0, np.abs(out[0][0]))).all()


@pytest.mark.parametrize("metal", [None, (9.0, 0.035)])
def test_nodes_by_one_warp_or_two(metal):
    """the K integrals of few matrices share 32 nodes between two warps, those of many do not: the same bits"""
    import caps_gb300 as cg
    c = cg.Caps(30e-6, 1e-6, ldim=60)
    if metal:
        c.set_drude(*metal)
    c.set_precision(cg.PREC_MIXED)
    xi, m = np.linspace(1.0, 40.0, 500), np.arange(500) % 7
    many, status = c.logdetD_batch(xi, m)
    assert (status < 16).all()
    for k in (0, 3, 250, 499):
        one, _ = c.logdetD_batch(xi[k:k + 1], m[k:k + 1])
        assert one[0] == many[k]
