"""FP64 products of entries over many decades, element by element: the error is relative to sum |a||b|, not to the
largest entries of the row and the column.

Bound.  An element comes from slices when the sum of its leading bytes' products is at least 16 sqrt(K); a byte
may round a magnitude up to twofold, so the product X of the two maxima's powers of two is at most 2^16 2 /
(16 sqrt(K)) = 2^13 / sqrt(K) times sum |a||b|.  The two roundings of a term have an rms of 2^-56.3 X each; eight
sigma over K independent terms: 2^-52.8 sqrt(K) X < 2^-39 of sum |a||b|.  NumPy's reference adds K 2^-52."""
import ctypes as C

import numpy as np
import pytest

import qrochet  # noqa: F401
from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu


def zgemm(opA, opB, A, B, M, N, K, dk=None):
    A, B = np.asfortranarray(A), np.asfortranarray(B)
    out = np.full((M, N), np.nan, dtype=np.complex128, order="F")
    one, zero, ms = np.array([1.0, 0.0]), np.zeros(2), C.c_double()
    _lib.check(_lib.lib().qr_test_zgemm(opA, opB, M, N, K, _lib.dptr(one), _lib.dptr(A), A.shape[0], _lib.dptr(B),
                                        B.shape[0], _lib.dptr(zero), _lib.dptr(out), M,
                                        None if dk is None else _lib.dptr(dk), 1, C.byref(ms)))
    return out


def wide(g, kind, *shape):
    z = R.complex_gaussian(g, shape)
    if kind == "lognormal":
        return z * np.exp(6 * g.standard_normal(shape))
    if kind == "decades":
        return z * 10.0 ** (-12 * g.random(shape))
    if kind == "blocks":  # large and small blocks, and zeros
        m = np.array([[1.0, 1e-14], [0.0, 1e-7]])
        return z * np.kron(m, np.ones(((shape[0] + 1) // 2, (shape[1] + 1) // 2)))[:shape[0], :shape[1]]
    return z * (g.random(shape) < 0.02)  # sparse


# one tile and several, ragged tiles, K split over clusters of 2 to 8 and not, few rows or columns
@pytest.mark.parametrize("M,N,K", [(128, 192, 64), (65, 130, 200), (64, 64, 512), (300, 17, 400), (3, 600, 1000),
                                   (129, 63, 2049)])
@pytest.mark.parametrize("kind", ["lognormal", "decades", "blocks", "sparse"])
def test_error_relative_to_the_terms(kind, M, N, K):
    g = R.rng(M + N + K)
    A, B = wide(g, kind, M, K), wide(g, kind, K, N)
    got = zgemm(0, 0, A, B, M, N, K)
    assert np.all(np.abs(got - A @ B) <= (2.0 ** -39 + K * 2.0 ** -52) * (np.abs(A) @ np.abs(B)))


@pytest.mark.parametrize("opA", [0, 1, 2, 3])
@pytest.mark.parametrize("opB", [0, 1, 2, 3])
def test_orders_with_a_diagonal(opA, opB):
    M, N, K = 130, 95, 150
    g = R.rng(7 + opA + 4 * opB)
    ops = {0: lambda x: x, 1: lambda x: x.T, 2: lambda x: x.conj().T, 3: lambda x: x.conj()}
    A, B, dk = wide(g, "lognormal", M, K), wide(g, "lognormal", K, N), 10.0 ** (-8 * g.random(K))
    got = zgemm(opA, opB, ops[opA](A), ops[opB](B), M, N, K, dk)
    A = A * dk[None, :]
    assert np.all(np.abs(got - A @ B) <= (2.0 ** -39 + K * 2.0 ** -52) * (np.abs(A) @ np.abs(B)))


def test_rows_whose_largest_entry_stands_out():
    """R of a QR times a site: the products that lie 2^-56 below the maxima count where a row's maximum is sixteen
    times the rest.  The rms error stays under 2^-53 sqrt(K) / 4, a fraction of what K roundings of a sum make."""
    K, N = 256, 64
    g = R.rng(77)
    A, B = np.triu(R.complex_gaussian(g, (K, K)) + 16 * np.eye(K)), R.complex_gaussian(g, (K, N))
    ref = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    err = np.linalg.norm((zgemm(0, 0, A, B, K, N, K) - ref).astype(complex)) / np.linalg.norm(ref.astype(complex))
    assert err <= 2.0 ** -53 * np.sqrt(K) / 4
