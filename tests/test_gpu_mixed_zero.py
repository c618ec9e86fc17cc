"""Mixed form: trailing updates without the image blocks that are zero.  Sizes at the ends of 64-row blocks, of
128-row tiles and of panels of 512 columns (dimension 2 ldim), matrices from full to almost empty factors, against the
FP64 form; bar: the mixed form's 5e-8 max(1, |x|) of the suite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ldim", [31, 32, 33, 64, 65, 96, 128, 160, 256, 257, 289, 320, 513, 600])
@pytest.mark.parametrize("rl", [8.0, 60.0])
def test_against_fp64(ldim, rl):
    import caps_gb300 as cg
    xi = np.array([0.02, 0.3, 1.5, 5.0, 0.1]) * (1 + rl) / 2
    m = np.array([0, 1, 2, 1, 30])
    out = []
    for prec in (cg.PREC_FP64, cg.PREC_MIXED):
        c = cg.Caps(rl * 1e-6, 1e-6, ldim=ldim)
        c.set_drude(9.0, 0.035)
        c.set_precision(prec)
        out.append(c.logdetD_batch(xi, m))
    assert (out[0][1] < 16).all() and (out[1][1] < 16).all()
    assert (np.abs(out[0][0] - out[1][0]) <= 5e-8 * np.maximum(1.0, np.abs(out[0][0]))).all()
