"""Sphere-sphere log det(1 - M^2): the fixed-point square at the sizes where its 64-row blocks and pairs of blocks
end, from frequencies where M is near 1 down to those where the trace and Mercator rules decide.

Reference: sum of log(1 - w^2) over the eigenvalues of the oracle's M.  Tolerance: M is good to 1e-13
relative and 1 - M^2 carries 2^-54 per entry, 2 n 2^-54 < 3e-14 in the log det for n <= 280, both as in the tests of
the factorisation; a Mercator result is good to 1e-8 by its rule, a trace result (below 1e-8) to its
square."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
R, L = 40e-6, 1e-6


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("ldim", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 140])
def test_sizes(ldim, mixed):
    import caps_gb300 as cg
    from oracle import binding as ob
    c = cg.Caps(R, L, ldim=ldim, detalg=cg.DETALG_LU)
    if mixed:
        c.set_precision(cg.PREC_MIXED)
    scale = (1 + R / L) / 2
    xi = np.array([0.05, 1.0, 0.3, 3.0, 5.5, 12.0, 60.0]) * scale
    m = np.array([0, 0, 3, 1, 2, 1, 5])
    got, status = c.logdetD2_batch(xi, m)
    assert (status < 16).all()
    for x, mm, v, st in zip(xi, m, got, status):
        M = ob.M_dense(R, L, ldim, x, int(mm))
        want = np.sum(np.log1p(-np.linalg.eigvalsh(M) ** 2))
        rel = {1: 1e-8, 2: 1e-8, 3: 5e-8 if mixed else 1e-10}[int(st)]
        assert abs(v - want) <= rel * abs(want) + (5e-8 if mixed and st == 3 else 3e-14 if st == 3 else 1e-16), (x, mm, st, v, want)
