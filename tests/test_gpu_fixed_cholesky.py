"""The fixed-point Cholesky of the FP64 form at the sizes where its tiles end: the 16-column
sub-panels and 64-column blocks of the diagonal kernel, pairs of 64-row blocks (odd and even
counts), a last block of one row, several column chunks per CTA.

The cylinder-plane determinant takes any dimension n = lmax, so it covers odd sizes; the oracle
restates it in FP64 (its LU and the library agree to a few units of rounding).  Tolerance: an
entry carries 2^-54 per factor and the log det sums 2 n of them with A^-1 of norm below 10^2, so
the error stays below 2 n 10^2 2^-54 < 2e-11 for the largest n here; 1e-12 max(1, |x|) + 1e-14 n
is inside that and far above what FP64 LU itself loses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 63, 64, 65, 80, 127, 128, 129, 191, 192, 193, 257, 321, 449])
@pytest.mark.parametrize("boundary", ["D", "N"])
def test_dimensions(n, boundary):
    import caps_gb300 as cg
    from oracle import binding as ob
    R, d = 30e-6, 1e-6
    q = np.array([0.01, 0.4, 3.0]) / (2 * d)
    got = cg.capc_logdet(R, d, q, boundary, n, "LU")
    for x, v in zip(q, got):
        want = ob.lib.oracle_capc_logdet(R, d, n, float(x), boundary.encode(), 0)
        assert abs(v - want) <= 1e-12 * max(1.0, abs(want)) + 1e-14 * n, (n, x, v, want)


@pytest.mark.parametrize("count", [1, 5, 40])
def test_batches(count):
    """results do not depend on the batch: chunks of one and of several column blocks per CTA"""
    import caps_gb300 as cg
    c = cg.Caps(60e-6, 1e-6, ldim=430)
    xi = np.linspace(5.0, 60.0, count)
    got, status = c.logdetD_batch(xi, np.full(count, 2))
    assert (status < 16).all()
    for k in {0, count // 2, count - 1}:
        assert got[k] == c.logdetD(xi[k], 2)


@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e-8, 1e-14])
def test_small_entries(scale):
    """matrices whose factor has whole blocks of zero digits (they are skipped), down to M below the last
    digit: high frequencies, against the trace or LU of the oracle's M (its own log det takes the Mercator
    shortcut here, good to 1e-8 only) relative to the value"""
    import caps_gb300 as cg
    from oracle import binding as ob
    R, L, ldim = 40e-6, 1e-6, 150
    c = cg.Caps(R, L, ldim=ldim, detalg=cg.DETALG_HODLR)
    # log det falls like e^{-2 xi L/c}: the decay that scales it by `scale`
    xi = (1 + R / L) / 2 * (0.5 - np.log(scale))
    got, status = c.logdetD_batch([xi, xi, xi], [0, 1, 4])
    assert (status < 16).all()
    for m, v in zip((0, 1, 4), got):
        M = ob.M_dense(R, L, ldim, xi, m)
        tr = np.trace(M)
        want = -tr if tr < 1e-8 else np.linalg.slogdet(np.eye(2 * ldim) - M)[1]
        assert abs(v - want) <= 1e-10 * abs(want) + 3e-14, (xi, m, v, want)


@pytest.mark.parametrize("ldim", [255, 256, 257, 288, 330])
@pytest.mark.parametrize("count", [1, 3, 170])
def test_updates_beside_panels(ldim, count):
    """both sides of the dimension (512) from which the rest of an update runs beside the next panel, for few and for
    many matrices, against LU of the oracle's M; the bar of the suite"""
    import caps_gb300 as cg
    from oracle import binding as ob
    R, L = 45e-6, 1e-6
    c = cg.Caps(R, L, ldim=ldim)
    xi = np.linspace(0.5, 30.0, count)
    got, status = c.logdetD_batch(xi, np.full(count, 1))
    assert (status < 16).all()
    for k in {0, count // 3, count - 1}:
        M = ob.M_dense(R, L, ldim, float(xi[k]), 1)
        want = np.linalg.slogdet(np.eye(2 * ldim) - M)[1]
        assert abs(got[k] - want) <= 1e-10 * max(1.0, abs(want)), (k, got[k], want)
        assert got[k] == c.logdetD(xi[k], 1)
