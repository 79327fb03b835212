"""A pair of equal singular values that the refinement rotates by a listed double-float sweep: the other columns
come out at FP64 accuracy all the same.

The matrix is diagonal but for one coupling below the FP32 sweeps' threshold, so a singular value is one entry:
its square, the sum and the root round to 2 eps at most; 4 eps of the largest is the bound (48 bits are 16)."""
import ctypes as C

import numpy as np
import pytest

import qrochet  # noqa: F401
from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [130, 200, 301, 600])
def test_singular_values_of_a_nearly_diagonal_matrix(k):
    s = np.sort(1 + R.rng(k).random(k))[::-1].copy()
    h = k // 2
    s[h + 1] = s[h]
    A = np.asfortranarray(np.diag(s).astype(np.complex128))
    A[h, h + 1] = 1e-7
    t = 0.5e-7  # [[d, 2 t], [0, d]]: sqrt(d^2 + t^2) +- t
    s[h], s[h + 1] = np.hypot(s[h], t) + t, np.hypot(s[h], t) - t
    U, Vh = np.empty((k, k), dtype=np.complex128, order="F"), np.empty((k, k), dtype=np.complex128, order="F")
    S, ms = np.empty(k), C.c_double()
    _lib.check(_lib.lib().qr_test_svd(0, k, k, _lib.dptr(A), _lib.dptr(U), _lib.dptr(S), _lib.dptr(Vh), C.byref(ms)))
    assert np.max(np.abs(S - np.sort(s)[::-1])) <= 4 * np.finfo(float).eps * s[0]
