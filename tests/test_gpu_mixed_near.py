"""Mixed form: diagonal blocks on both sides of |S| = 2^-13, below which the factor is taken to second order, against
the FP64 form.  Tolerance: FP32 entries of M (6e-8 relative, of either sign) average out to 1e-8 of the log det
in the suite's matrices; 5e-8 of the value, and 1e-14 for values near the trace rule's line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ldim", [5, 32, 33, 150])
@pytest.mark.parametrize("bits", [4, 8, 11, 12, 13, 14, 15, 18, 22])
def test_lines(ldim, bits):
    import caps_gb300 as cg
    R, L = 40e-6, 1e-6
    xi = (1 + R / L) / 2 * bits * np.log(2.0)
    out = []
    for prec in (cg.PREC_FP64, cg.PREC_MIXED):
        c = cg.Caps(R, L, ldim=ldim)
        c.set_precision(prec)
        out.append(c.logdetD_batch([xi, xi, xi], [0, 1, 4]))
    assert (out[0][1] < 16).all() and (out[1][1] < 16).all()
    assert (np.abs(out[0][0] - out[1][0]) <= 5e-8 * np.abs(out[0][0]) + 1e-14).all()
