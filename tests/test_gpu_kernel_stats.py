"""The byte counter of the mixed form's updates: cleared between batches, and before the next one adds to it, so that every
batch of the same matrices counts the same bytes (whole 128 x 64 tiles of S, read and written in FP32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_same_bytes_every_time():
    import caps_gb300 as cg
    c = cg.Caps(60e-6, 1e-6, ldim=420)
    c.set_drude(9.0, 0.035)
    c.set_precision(cg.PREC_MIXED)
    xi, m = np.repeat(np.linspace(8.0, 60.0, 6), 4), np.tile(np.arange(4), 6)
    c.logdetD_batch(xi, m)
    seen = set()
    try:
        for _ in range(20):
            cg.kernel_timing(True)
            for k in (1, 2):  # cleared when it is switched on, and by each batch
                c.logdetD_batch(xi, m)
                ms, nbytes, launches = cg.kernel_stats(0)
                assert ms > 0 and launches > 0 and nbytes > 0 and nbytes % (k * 128 * 64 * 8) == 0
                seen.add(nbytes / k)
    finally:
        cg.kernel_timing(False)
    assert len(seen) == 1, seen
