"""Batched FP64 products on exact slices whose workspace holds a part of the batch only, or none of it: runs of
entries give the bits of one run over the whole batch (the guarded product, whose last accumulator rounds, the same
values); without memory the CUDA cores give the product."""
import ctypes as C

import numpy as np
import pytest

import qrochet  # noqa: F401
from qrochet import _lib
from qrochet import random as R

pytestmark = pytest.mark.gpu

ROOM = 1 << 30


def batched(A, B, room, opA=0, guard=0):
    batch, N, M = A.shape[0], B.shape[-1], A.shape[1] if opA == 0 else A.shape[2]
    K = B.shape[-2]
    fa = np.ascontiguousarray(np.swapaxes(A, 1, 2))  # column-major matrices, one after another
    fb = np.ascontiguousarray(np.swapaxes(B, -1, -2))
    out, ms = np.empty((batch, N, M), dtype=np.complex128), C.c_double()
    _lib.check(_lib.lib().qr_test_zgemm_oz(opA, 0, M, N, K, batch, int(B.ndim == 2), _lib.dptr(fa), A.shape[1],
                                           _lib.dptr(fb), K, _lib.dptr(out), guard, room, C.byref(ms)))
    return np.swapaxes(out, 1, 2)


# bytes of an entry: 14 per element of A's planes (2 M' x 2 K', M' and K' whole tiles), about 28 K' N' for B
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("batch,M,N,K", [(1, 70, 65, 48), (5, 70, 65, 48), (7, 64, 64, 16), (9, 130, 3, 200)])
def test_runs_of_a_batch(shared, batch, M, N, K):
    g = R.rng(batch * M + N)
    A, B = R.complex_gaussian(g, (batch, M, K)), R.complex_gaussian(g, (K, N) if shared else (batch, K, N))
    whole = batched(A, B, ROOM)
    up = lambda x, q: (x + q - 1) // q * q  # noqa: E731
    entry = 7 * 2 * 2 * up(M, 64) * 2 * up(K, 16) + 4 * M
    b = 7 * 2 * up(N, 64) * 2 * up(K, 16) + 4 * (N + K)
    for room in (1, 2 * entry + (b if shared else 2 * b), 3 * entry + (b if shared else 3 * b)):
        assert np.array_equal(batched(A, B, room), whole)
    ref = A @ B
    bound = K * 2.0 ** -50 * np.max(np.abs(A)) * np.max(np.abs(B))
    assert np.max(np.abs(whole - ref)) <= bound
    for room in (0, 1, 3 * entry + (b if shared else 3 * b), ROOM):
        assert np.max(np.abs(batched(A, B, room, guard=1) - ref)) <= bound


def test_transposed_operand_in_runs():
    g = R.rng(8)
    A, B = R.complex_gaussian(g, (4, 90, 66)), R.complex_gaussian(g, (90, 40))
    whole = batched(A, B, ROOM, opA=2)
    assert np.array_equal(batched(A, B, 1, opA=2), whole)
    ref = np.conj(np.swapaxes(A, 1, 2)) @ B
    assert np.max(np.abs(whole - ref)) <= 90 * 2.0 ** -50 * np.max(np.abs(A)) * np.max(np.abs(B))
