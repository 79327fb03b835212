"""The order in which the SVD ranks column norms, on the CPU: a permutation for any keys (gathers and scatters
go through it), descending, ties by index, NaN first."""
import ctypes as C

import numpy as np
import pytest

from qrochet import _lib

NAN, INF = float("nan"), float("inf")


@pytest.mark.parametrize("keys", [[], [1.0], [NAN], [2.0, 2.0, 2.0], [NAN] * 5, [1.0, NAN, 3.0, NAN, 3.0, 0.0],
                                  [INF, NAN, INF, 0.0, -0.0, 5.0], [-1.0, 2.0, -INF, -3.0, NAN, 0.0], [0.0] * 7 + [NAN], [NAN] + [1.0] * 40])
def test_ranks_are_a_permutation(keys):
    k = np.array(keys, dtype=np.float64)
    perm = np.full(k.size + 1, -1, dtype=np.int32)
    _lib.check(_lib.lib().qr_test_rank_order(_lib.dptr(k), k.size, perm.ctypes.data_as(C.POINTER(C.c_int))))
    assert perm[-1] == -1
    want = sorted(range(k.size), key=lambda i: (not np.isnan(k[i]), 0.0 if np.isnan(k[i]) else -k[i], i))
    assert list(perm[:-1]) == want
