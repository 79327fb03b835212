"""Non-finite data ends in a status, never in a gather through an unwritten index: the SVD on each of its
routes (one cluster, FP32 sweeps in a cluster, grid sweeps, QR first or not), and one request of a batch."""
import numpy as np
import pytest

import qrochet as Q
from qrochet import _lib
from qrochet import random as R
from qrochet import serve as S
from qrochet.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("chi", [10, 32, 100])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_gate_on_a_non_finite_site(precision, chi, bad):
    g = R.rng(chi)
    a = R.complex_gaussian(g, (2, chi, chi))
    b = R.complex_gaussian(g, (2, chi, chi))
    ends = np.ones((2, chi), dtype=np.complex128)
    a[1, chi // 2, 3] = bad
    psi = Q.MPS([ends, a, b, ends])
    psi.set_precision(precision)
    with pytest.raises(_lib.GPUError, match="non-finite|converge|unitary"):
        Q.evolve_(psi, Q.gate_from_matrix(R.haar_unitary(g, 4), [2, 3]), threshold=1e-10, maxdim=chi)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_non_finite_gate_spoils_its_request_only(precision):
    g = R.rng(5)
    reqs = [S.random_request(g, n_range=(10, 10), depth_range=(8, 8), chi_choices=(32,), nobs=2) for _ in range(3)]
    site, u = reqs[1].gates[len(reqs[1].gates) // 2]
    u = np.array(u)
    u[2, 1] = np.nan
    reqs[1].gates[len(reqs[1].gates) // 2] = (site, u)
    with Batch(precision=precision) as b:
        ids = [b.add(r) for r in reqs]
        b.run()
        assert [b.result(i)["status"] == 0 for i in ids] == [True, False, True]
        got = [b.values(ids[0]), b.values(ids[2])]
    with Batch(precision=precision) as b:
        ids = [b.add(reqs[0]), b.add(reqs[2])]
        b.run()
        assert all(np.array_equal(x, b.values(i)) for x, i in zip(got, ids))
