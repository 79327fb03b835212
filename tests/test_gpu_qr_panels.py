"""The blocked Householder QR against its defining properties: panels of 32 columns in clusters of up to 16
CTAs with at least 16 rows each, block reflectors as products, the cooperative kernel beyond 6144 rows.

Bounds: Householder factors are backward stable, ||A - QR|| and ||Q^H Q - I|| within a modest multiple of
sqrt(m) n eps; 20 sqrt(m) eps relative to the largest column norm per entry covers the sizes below."""
import ctypes as C

import numpy as np
import pytest

from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu


def qr(A):
    m, n = A.shape
    k = min(m, n)
    A = np.asfortranarray(A, dtype=np.complex128)
    Q, Rm = np.empty((m, k), dtype=np.complex128, order="F"), np.empty((k, n), dtype=np.complex128, order="F")
    ms = C.c_double()
    _lib.check(_lib.lib().qr_test_qr(m, n, _lib.dptr(A), _lib.dptr(Q), _lib.dptr(Rm), C.byref(ms)))
    return Q, Rm


def check(A):
    Q, Rm = qr(A)
    m = A.shape[0]
    tol = 20 * np.sqrt(m) * 2.0 ** -52
    scale = np.max(np.linalg.norm(A, axis=0))
    assert np.max(np.abs(Q @ Rm - A)) <= tol * scale
    assert np.max(np.abs(Q.conj().T @ Q - np.eye(Q.shape[1]))) <= tol
    assert np.all(np.tril(Rm, -1) == 0)
    assert np.max(np.abs(np.diag(Rm).imag)) <= tol * scale  # LAPACK's real diagonal
    return Q, Rm


@pytest.mark.parametrize("m,n", [(1, 1), (3, 7), (16, 16), (17, 5), (31, 40), (32, 32), (33, 32), (65, 64), (97, 130),
                                 (256, 31), (257, 96), (300, 257), (1000, 129), (129, 1000), (4100, 33), (6144, 8),
                                 (6145, 8)])
def test_shapes(m, n):
    A = R.complex_gaussian(R.rng(m * 1009 + n), (m, n))
    Q, Rm = check(A)
    q, r = np.linalg.qr(A)
    # the same convention: the factors themselves agree (Gaussian columns are far from dependent when m > n)
    if m > 2 * n:
        assert np.max(np.abs(Rm - r)) <= 1e-12 * np.max(np.abs(r))
        assert np.max(np.abs(Q - q)) <= 1e-12


@pytest.mark.parametrize("kind", ["dependent", "zero columns", "triangular", "graded", "tiny", "huge"])
def test_matrices(kind):
    g = R.rng(17)
    A = R.complex_gaussian(g, (200, 90))
    if kind == "dependent":
        A[:, 40] = A[:, 3] + 2 * A[:, 39]
        A[:, 70:80] = A[:, 10:20]
    elif kind == "zero columns":
        A[:, [0, 31, 32, 89]] = 0
    elif kind == "triangular":  # nothing to reflect: tau = 0 where the diagonal is real
        A = np.triu(A)
        np.fill_diagonal(A, np.abs(np.diag(A)))
    elif kind == "graded":
        A = A * 10.0 ** (-12 * np.arange(90) / 90)
    elif kind == "tiny":
        A = A * 1e-140
    else:
        A = A * 1e140
    check(A)
