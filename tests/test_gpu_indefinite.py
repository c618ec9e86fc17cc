"""The fixed-point Cholesky of matrices that are not positive definite: integers of a fixed range wrap there, and every one
has to end as a pivot that is not positive (NaN, ST_ERR_PIVOT), wherever the matrix first leaves the range: an
entry beyond it, a row of the factor beyond its diagonal, a 64 x 64 block or the panels below, one step or a sum of
many.  And matrices close to those bounds that are positive definite still give their log det.

The factorisation is called on matrices made here, through tests/native/fixed_cholesky.cu."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PIVOT = 16


@pytest.fixture(scope="module")
def factor(tmp_path_factory):
    import caps_gb300 as cg
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("native") / "fixed_cholesky.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-w", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(ROOT, "caps_gb300", "csrc"), os.path.join(ROOT, "tests", "native", "fixed_cholesky.cu"),
                    "-o", so, cg.LIB_PATH, "-Xlinker", "-rpath," + os.path.dirname(cg.LIB_PATH)], check=True)
    lib = C.CDLL(so)

    def call(A):
        A = np.ascontiguousarray(A, dtype=np.float64)  # symmetric: rows or columns first
        k, n, _ = A.shape
        ld, st = np.empty(k), np.empty(k, dtype=np.int32)
        lib.fixed_logdet(A.ctypes.data_as(C.c_void_p), n, k, ld.ctypes.data_as(C.c_void_p), st.ctypes.data_as(C.c_void_p))
        return ld, st
    return call


def refused(factor, A):
    ld, st = factor(A)
    assert np.isnan(ld).all() and (st & PIVOT).all(), (ld, st)


@pytest.mark.parametrize("n", [2, 64, 65, 130, 200])
@pytest.mark.parametrize("entry", [1.001, 1.5, 2.0, 2.83, 3.9, 3.9999, 4.0, 4.5, 5.65, 7.0, 8.0, 16.0, 1e3, 1e19, 1e300, np.inf, np.nan])
def test_one_entry(factor, n, entry):
    """the identity with one entry off the diagonal that is larger than it, in a block and between blocks"""
    mats = []
    for i, j in {(n - 1, 0), (n // 2, max(n // 2 - 1, 0)), (n - 1, n // 3)}:
        for s in (entry, -entry):
            A = np.eye(n)
            A[i, j] = A[j, i] = s
            mats.append(A)
    refused(factor, np.array(mats))


@pytest.mark.parametrize("n", [65, 130, 257])
@pytest.mark.parametrize("small", [1e-1, 1e-2, 1e-4, 1e-6, 1e-9])
def test_small_pivot(factor, n, small):
    """an entry beyond sqrt(A_ii A_jj) by a small A_jj: the row of the factor is as large as 1 / sqrt(A_jj)"""
    mats = []
    for i, j in ((n - 1, 0), (n - 1, 40), (20, 3)):
        for x in (1.01, 1.9, 2.0, 3.0, 4.0, 4.1, 8.0, 16.0, 30.0):  # entry / sqrt(A_jj)
            A = np.eye(n)
            A[j, j] = small
            A[i, j] = A[j, i] = min(x * np.sqrt(small), 1.99)
            mats.append(A)
    refused(factor, np.array([A for A in mats if np.linalg.eigvalsh(A)[0] < 0]))


@pytest.mark.parametrize("n", [64, 65, 130, 200, 330])
@pytest.mark.parametrize("norm2", [1.01, 2.0, 3.0, 4.0, 7.9, 8.0, 9.0, 15.9, 16.0, 17.0, 32.0, 64.0])
def test_row_of_many(factor, n, norm2):
    """a row whose entries are all small, but whose squares add up beyond its diagonal: in one panel, over all panels"""
    mats = []
    for cols in (range(n - 1), range(min(63, n - 1)), range(max(n - 40, 0), n - 1)):
        c = np.array(list(cols))
        A = np.eye(n)
        A[n - 1, c] = A[c, n - 1] = np.sqrt(norm2 / len(c))
        mats.append(A)
    refused(factor, np.array(mats))


@pytest.mark.parametrize("n", [48, 90, 150, 290])
def test_random(factor, n):
    """random symmetric matrices of unit diagonal scale with one or many negative eigenvalues"""
    r = np.random.default_rng(n)
    mats = []
    for k in range(24):
        q = np.linalg.qr(r.standard_normal((n, n)))[0]
        w = r.uniform(0.05, 1.0, n)
        w[:1 + k * n // 48] *= -10.0 ** r.uniform(-3, 1)
        A = (q * w) @ q.T
        mats.append((A + A.T) / 2 / max(1.0, np.abs(np.diag(A)).max()))
    refused(factor, np.array(mats))


@pytest.mark.parametrize("n", [64, 65, 100, 128, 190, 300])
def test_close_to_the_bounds(factor, n):
    """diagonals up to 2, rows nearly parallel (their squares reach the diagonal), W up to 2^12 (its exponent is not zero),
    and a scaled matrix: condition numbers below 10^5, so 2^-54 per entry leaves 1e-16 10^5 n < 1e-8"""
    r = np.random.default_rng(n)
    mats = []
    for d in (1.0, 1.99, 1.9999, 7.0, 1e6):
        for rho in (0.0, 0.9, 0.99, 0.999):
            A = d * ((1 - rho) * np.eye(n) + rho)
            mats.append(A)
            s = 1 - 2 * (r.random(n) < 0.5)
            mats.append(A * np.outer(s, s))
        q = np.linalg.qr(r.standard_normal((n, n)))[0]
        A = (q * np.exp(r.uniform(-8, 0, n))) @ q.T
        mats.append(d * (A + A.T) / 2 / np.diag(A).max())
        A = np.eye(n) * d  # a 2 x 2 with eigenvalues of 10^-4 d
        A[n - 1, 0] = A[0, n - 1] = d * (1 - 1e-4)
        mats.append(A)
    A = np.array(mats)
    ld, st = factor(A)
    want = np.linalg.slogdet(A)[1]
    assert (st < 16).all(), st
    assert (np.abs(ld - want) <= 1e-8 * np.maximum(1, np.abs(want))).all(), (ld - want)
