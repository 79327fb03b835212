"""The operator mixing of an MPO expectation value over sparse site tensors: coefficients 1, i, -1, -i, real and
complex, bond dimensions around its blocks of 32 to 256 rows, and a site whose channels do not fit its staging.
Against a site by site contraction in numpy at 1e-11 of <psi|psi> |W|."""
import numpy as np
import pytest

import qrochet as Q
from qrochet import random as R

pytestmark = pytest.mark.gpu

COEFS = np.array([1, 1j, -1, -1j, 0.75, -2.5, 0.3 - 0.4j, 1 + 1j])


def _mpo(g, bonds):
    """Site tensors (o, i, l, r) with about a quarter of the entries set."""
    out = []
    for l, r in zip([1] + bonds, bonds + [1]):
        a = np.where(g.random((2, 2, l, r)) < 0.25, COEFS[g.integers(0, 8, (2, 2, l, r))], 0)
        a[0, 0, 0, 0] = a[1, 1, 0, 0] = 1  # the identity string survives
        out.append(a)
    return out


def _sweep(sites, ws):
    """<psi|W|psi> with site arrays (o, l, r) and W (o, i, l, r)."""
    e = np.ones((1, 1, 1), dtype=np.complex128)  # ket, channel, bra
    for a, w in zip(sites, ws):
        x = np.tensordot(e, a, (0, 1))                       # w b i a'
        x = np.tensordot(w, x, ((1, 2), (2, 0)))             # o w' b a'
        e = np.transpose(np.tensordot(x, a.conj(), ((0, 2), (0, 1))), (1, 0, 2))
    return e[0, 0, 0]


@pytest.mark.parametrize("chi,bonds", [(1, [2, 3, 2]), (5, [3, 5, 4]), (31, [5, 5, 5]), (33, [4, 8, 3]), (130, [5, 2, 5]),
                                       (257, [3, 5, 3]), (6, [49, 1, 2]), (9, [2, 60, 2])])
def test_sparse_mixing(chi, bonds):
    g = R.rng(chi)
    n = len(bonds) + 1
    full = []
    for i in range(n):
        cl, cr = (1 if i == 0 else chi), (1 if i == n - 1 else chi)
        full.append(R.complex_gaussian(g, (2, cl, cr)) / np.sqrt(2 * cl))
    ws = _mpo(g, bonds)
    psi = Q.MPS([full[0][:, 0, :], *full[1:-1], full[-1][:, :, 0]])
    H = Q.MPO([ws[0][:, :, 0, :], *ws[1:-1], ws[-1][:, :, :, 0]])
    one = [np.eye(2).reshape(2, 2, 1, 1)] * n
    scale = abs(_sweep(full, one)) * np.prod([np.linalg.norm(w) for w in ws])
    assert abs(Q.mpo_expect(psi, H) - _sweep(full, ws)) <= 1e-11 * scale
