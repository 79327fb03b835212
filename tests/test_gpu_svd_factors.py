"""The SVD's factors over spectra that spread over three decades: orthonormal and exact at the level that rounding
leaves, not only at the tolerance of the rotation test.

Bound.  U's columns are those of B = A V, which carry the rounding of k-term sums of A's largest entries, sqrt(k)
eps sigma_max, and are then made orthogonal; V's are products of unitary corrections; both keep sqrt(k) eps with a
factor below 4.  A - U S V^H adds the couplings that are left, at most a sixteenth of the tolerance sqrt(k) eps
sigma_max each, k of them to a column in random sign: k / 16 eps sigma_max.  Together 4 sqrt(k) + k / 16 in eps; the
factors are held to twice that."""
import ctypes as C

import numpy as np
import pytest

import qrochet  # noqa: F401
from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu


# one cluster (up to 32 columns), and the refinement on the tensor cores, in FP64
@pytest.mark.parametrize("n", [4, 9, 12, 16, 24, 32, 48, 128, 300])
@pytest.mark.parametrize("kind", ["gaussian", "linear", "decades"])
def test_orthonormal_to_rounding(n, kind):
    worst = np.zeros(3)
    for seed in range(6 if n <= 32 else 1):
        g = R.rng(1000 * n + seed)
        A = R.complex_gaussian(g, (n, n))
        if kind != "gaussian":
            u, _ = np.linalg.qr(A)
            v, _ = np.linalg.qr(R.complex_gaussian(g, (n, n)))
            A = (u * (np.linspace(1, 0.01, n) if kind == "linear" else np.logspace(0, -2.9, n))) @ v.conj().T
        A = np.asfortranarray(A)
        U, Vh = np.empty((n, n), dtype=np.complex128, order="F"), np.empty((n, n), dtype=np.complex128, order="F")
        S, ms = np.empty(n), C.c_double()
        _lib.check(_lib.lib().qr_test_svd(0, n, n, _lib.dptr(A), _lib.dptr(U), _lib.dptr(S), _lib.dptr(Vh),
                                          C.byref(ms)))
        eye = np.eye(n)
        worst = np.maximum(worst, [np.linalg.norm(U.conj().T @ U - eye, 2), np.linalg.norm(Vh @ Vh.conj().T - eye, 2),
                                   np.linalg.norm((U * S) @ Vh - A, 2) / S[0]])
    assert np.all(worst <= 2 * (4 * np.sqrt(n) + n / 16) * np.finfo(float).eps)
