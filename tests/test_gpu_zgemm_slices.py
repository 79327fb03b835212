"""The FP64 GEMM on exact integer slices (tensor cores) and its small-product FP64 kernel, against NumPy.

Bound per element, from the slicing: an entry is held to 2^-55 of its scaled row (column) maximum, the
neglected slice products add 2^-51 of the maxima, four real products per complex one, K terms; with
op(B)'s rows equilibrated the maxima are max_k |A_ik| max_j |B_kj|: K 2^-50 of that, NumPy's own rounding
included."""
import ctypes as C

import numpy as np
import pytest

from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu

OPS = {0: lambda x: x, 1: lambda x: x.T, 2: lambda x: x.conj().T, 3: lambda x: x.conj()}


def zgemm(opA, opB, A, B, M, N, K, dk=None):
    A, B = np.asfortranarray(A), np.asfortranarray(B)
    out = np.full((M, N), np.nan, dtype=np.complex128, order="F")
    one, zero, ms = np.array([1.0, 0.0]), np.zeros(2), C.c_double()
    _lib.check(_lib.lib().qr_test_zgemm(opA, opB, M, N, K, _lib.dptr(one), _lib.dptr(A), A.shape[0], _lib.dptr(B),
                                        B.shape[0], _lib.dptr(zero), _lib.dptr(out), M,
                                        None if dk is None else _lib.dptr(dk), 1, C.byref(ms)))
    return out


def check(got, A, B):
    K = A.shape[1]
    a = np.max(np.abs(A) * np.max(np.abs(B), axis=1)[None, :], axis=1)
    assert np.all(np.abs(got - A @ B) <= K * 2.0 ** -50 * a[:, None])


# a tile is 64 x 64 (complex rows x columns), a stage 16 complex k, accumulators drain after 128 k, and K
# splits over clusters of up to 8; the last two sizes stay on the small-product kernel
@pytest.mark.parametrize("M,N,K", [(64, 64, 512), (65, 130, 193), (129, 63, 257), (1, 1700, 1000), (1500, 3, 401),
                                   (320, 320, 17), (200, 170, 128), (700, 640, 144), (64, 65, 2049), (40, 33, 70),
                                   (3, 5, 7)])
def test_sizes(M, N, K):
    g = R.rng(M + 31 * N + 1009 * K)
    A, B = R.complex_gaussian(g, (M, K)), R.complex_gaussian(g, (K, N))
    check(zgemm(0, 0, A, B, M, N, K), A, B)


@pytest.mark.parametrize("opA", [0, 1, 2, 3])
@pytest.mark.parametrize("opB", [0, 1, 2, 3])
def test_ops_with_diagonal(opA, opB):
    M, N, K = 130, 95, 150
    g = R.rng(7 + opA + 4 * opB)
    A, B, dk = R.complex_gaussian(g, (M, K)), R.complex_gaussian(g, (K, N)), g.random(K)
    check(zgemm(opA, opB, OPS[opA](A), OPS[opB](B), M, N, K, dk), A * dk[None, :], B)


@pytest.mark.parametrize("kind", ["positive", "constant", "graded", "tiny", "huge", "zero rows"])
def test_value_ranges(kind):
    M, N, K = 128, 160, 3000
    g = R.rng(99)
    A, B = R.complex_gaussian(g, (M, K)), R.complex_gaussian(g, (K, N))
    if kind == "positive":
        A, B = g.random((M, K)) + 1j * g.random((M, K)), g.random((K, N)) + 1j * g.random((K, N))
    elif kind == "constant":
        A, B = np.full((M, K), 0.7 + 0.3j), np.full((K, N), 1 / 3 + 0.9j)
    elif kind == "graded":  # Gamma-like against Lambda-like operands: every k contributes equally
        lam = 10.0 ** (-14 * np.arange(K) / K)
        A, B = A * lam, B / lam[:, None]
    elif kind == "tiny":
        A, B = A * 1e-150, B * 1e-140
    elif kind == "huge":
        A, B = A * 1e150, B * 1e150
    else:
        A[5], B[:, 7], B[11] = 0, 0, 0
    check(zgemm(0, 0, A, B, M, N, K), A, B)


def test_non_finite_entries_follow_the_plain_product():
    M, N, K = 100, 150, 200
    g = R.rng(3)
    A, B = R.complex_gaussian(g, (M, K)), R.complex_gaussian(g, (K, N))
    A[3, 5], B[7, 9] = np.inf, np.nan
    got = zgemm(0, 0, A, B, M, N, K)
    bad = np.zeros((M, N), dtype=bool)
    bad[3], bad[:, 9] = True, True
    assert np.array_equal(~np.isfinite(got), bad)
    A[3, 5], B[7, 9] = 0, 0
    ref = A @ B
    assert np.max(np.abs(got - ref)[~bad]) <= 1e-13 * np.max(np.abs(ref))
