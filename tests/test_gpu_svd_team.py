"""The SVD of one small matrix on one cluster: sizes around the limits of its blocks, lanes and dispatch, spectra
that need its second FP32 pass or full sweeps, and zeros, against LAPACK.  Tolerance 1e-12 of the largest singular
value (double-float products of up to 128 terms carry ~1e-14)."""
import ctypes as C

import numpy as np
import pytest

from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu


def svd(mode, A):
    A = np.asfortranarray(A, dtype=np.complex128)
    m, n = A.shape
    k = min(m, n)
    U, Vh = np.empty((m, k), dtype=np.complex128, order="F"), np.empty((k, n), dtype=np.complex128, order="F")
    S, ms = np.empty(k), C.c_double()
    _lib.check(_lib.lib().qr_test_svd(mode, m, n, _lib.dptr(A), _lib.dptr(U), _lib.dptr(S), _lib.dptr(Vh),
                                      C.byref(ms)))
    return U, S, Vh


def check(mode, A, tol=1e-12):
    U, S, Vh = svd(mode, A)
    ref = np.linalg.svd(A, compute_uv=False)
    eye = np.eye(S.size)
    assert np.max(np.abs(S - ref)) <= tol * ref[0]
    assert np.max(np.abs((U * S) @ Vh - A)) <= tol * ref[0]
    assert np.max(np.abs(U.conj().T @ U - eye)) <= tol
    assert np.max(np.abs(Vh @ Vh.conj().T - eye)) <= tol


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m,n", [(2, 2), (128, 2), (3, 7), (8, 8), (9, 12), (16, 16), (17, 17), (23, 128), (24, 31), (32, 32), (128, 32), (129, 32), (33, 33),
                                 (40, 39), (64, 65), (65, 100), (127, 127), (128, 128), (17, 129)])
def test_sizes(mode, m, n):
    check(mode, R.complex_gaussian(R.rng(m * 131 + n), (m, n)))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [8, 20, 32, 100, 128])
@pytest.mark.parametrize("kind", ["equal", "degenerate", "clusters", "decades", "steep", "rank"])
def test_spectra(mode, n, kind):
    g = R.rng(n)
    s = {"equal": np.ones(n), "degenerate": np.repeat([1.0, 0.5, 0.25, 0.1], n // 4),
         "clusters": np.concatenate([1 + 1e-7 * g.random(n // 2), 0.5 + 1e-10 * g.random(n - n // 2)]),
         "decades": np.logspace(0, -11, n), "steep": np.logspace(0, -100, n),
         "rank": np.where(np.arange(n) < n // 5, 1.0 + np.arange(n), 0.0)}[kind]
    u, _ = np.linalg.qr(R.complex_gaussian(g, (n, n)))
    v, _ = np.linalg.qr(R.complex_gaussian(g, (n, n)))
    check(mode, (u * np.sort(s)[::-1]) @ v.conj().T, 1e-11 if kind == "clusters" else 1e-12)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [20, 64])
def test_zeros(mode, n):
    U, S, Vh = svd(mode, np.zeros((n, n)))
    assert not S.any() and np.allclose(Vh @ Vh.conj().T, np.eye(n))
    A = np.zeros((n, n), dtype=np.complex128)
    A[3, 5] = 2.0 - 1.0j
    U, S, Vh = svd(mode, A)
    assert abs(S[0] - abs(A[3, 5])) < 1e-14 and not S[1:].any()
    assert np.max(np.abs((U * S) @ Vh - A)) < 1e-14
