"""The SVD's FP32 sweeps on Gram matrices and its finish by matrix products: sizes around the limits of their
launches, kept triplets, and spectra that steer it (degenerate and clustered values fall back to sweeps, graded ones restart on R^H).

Both precisions must give LAPACK's values and factors orthonormal and exact to rounding: 1e-12 relative to
sigma_max covers sqrt(512) eps with a factor 200; the clustered spectrum in mixed precision ends in
double-float sweeps (2^-44) and is held to 1e-11."""
import ctypes as C

import numpy as np
import pytest

import qrochet as Q
from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu


def svd(mode, A):
    A = np.asfortranarray(A, dtype=np.complex128)
    m, n = A.shape
    k = min(m, n)
    U = np.empty((m, k), dtype=np.complex128, order="F")
    Vh = np.empty((k, n), dtype=np.complex128, order="F")
    S, ms = np.empty(k), C.c_double()
    _lib.check(_lib.lib().qr_test_svd(mode, m, n, _lib.dptr(A), _lib.dptr(U), _lib.dptr(S), _lib.dptr(Vh),
                                      C.byref(ms)))
    return U, S, Vh


def check(mode, A, tol=1e-12):
    U, S, Vh = svd(mode, A)
    ref = np.linalg.svd(A, compute_uv=False)
    k = S.size
    assert np.max(np.abs(S - ref)) <= tol * ref[0]
    assert np.max(np.abs((U * S) @ Vh - A)) <= tol * ref[0]
    assert np.max(np.abs(U.conj().T @ U - np.eye(k))) <= tol
    assert np.max(np.abs(Vh @ Vh.conj().T - np.eye(k))) <= tol


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m,n", [(17, 17), (33, 90), (128, 128), (129, 128), (129, 129), (130, 300), (191, 191),
                                 (192, 192), (400, 193), (2049, 130), (513, 513),
                                 # FP32 sweeps: 8- and 16-column blocks, one CTA of 256 rows, clusters of 128-row
                                 # and 256-row CTAs with a ragged last one, odd block counts, rows beyond a cluster
                                 (256, 136), (257, 140), (385, 137), (897, 140), (1300, 161), (4096, 129), (4097, 129)])
def test_sizes(mode, m, n):
    check(mode, R.complex_gaussian(R.rng(m * 7 + n), (m, n)))


def _with_spectrum(g, n, s):
    u, _ = np.linalg.qr(R.complex_gaussian(g, (n, n)))
    v, _ = np.linalg.qr(R.complex_gaussian(g, (n, n)))
    return (u * s) @ v.conj().T


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [64, 200])
@pytest.mark.parametrize("kind", ["degenerate", "clusters", "pairs", "decades", "rank"])
def test_spectra(mode, n, kind):
    g = R.rng(n)
    s = {"degenerate": np.repeat([1.0, 0.5, 0.25, 0.1], n // 4),
         "clusters": np.concatenate([1 + 1e-7 * g.random(n // 2), 0.5 + 1e-10 * g.random(n - n // 2)]),
         "pairs": np.repeat(np.linspace(1, 0.2, n // 2), 2) * (1 + 1e-9 * g.random(n)),
         "decades": np.logspace(0, -11, n),
         "rank": np.where(np.arange(n) < n // 5, 1.0 + np.arange(n), 0.0)}[kind]
    check(mode, _with_spectrum(g, n, np.sort(s)[::-1]), 1e-11 if kind == "clusters" else 1e-12)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("chi,maxdim", [(40, 33), (100, 64), (150, 150)])
def test_kept_triplets_of_a_rank_deficient_block(precision, chi, maxdim):
    """theta of a gate with no entangling power has rank chi of 2 chi: the kept columns must not take up
    any of the noise columns behind them."""
    g = R.rng(chi)
    a = R.complex_gaussian(g, (2, chi, chi)) / np.sqrt(2 * chi)
    b = R.complex_gaussian(g, (2, chi, chi)) / np.sqrt(2 * chi)
    ends = np.ones((2, chi), dtype=np.complex128)
    psi = Q.MPS([ends, a, b, ends])
    psi.set_precision(precision)
    u = np.kron(R.haar_unitary(g, 2), R.haar_unitary(g, 2))
    Q.evolve_(psi, Q.gate_from_matrix(u, [2, 3]), threshold=1e-10, maxdim=maxdim)
    t = np.einsum("abcd,lcdr->labr", u.reshape(2, 2, 2, 2), np.einsum("alx,bxr->labr", a, b)).reshape(2 * chi, 2 * chi)
    uu, s, vv = np.linalg.svd(t)
    x, y = psi.site_array(2), psi.site_array(3)
    lam = psi.lambda_between(2, 3)
    assert lam.size == maxdim
    assert np.max(np.abs(lam - s[:maxdim])) <= 1e-12 * s[0]
    x = np.transpose(x, (1, 0, 2)).reshape(2 * chi, -1)
    y = np.transpose(y, (1, 0, 2)).reshape(-1, 2 * chi)
    ref = (uu[:, :maxdim] * s[:maxdim]) @ vv[:maxdim]
    gap = (s[maxdim - 1] - s[maxdim]) / s[0]
    assert np.max(np.abs((x * lam) @ y - ref)) <= 1e-12 * s[0] / min(1.0, gap)
    assert np.max(np.abs(x.conj().T @ x - np.eye(maxdim))) <= 1e-12
    assert np.max(np.abs(y @ y.conj().T - np.eye(maxdim))) <= 1e-12
