"""The batched engine's cluster kernels at bond dimensions that do not divide over a cluster's CTAs: Pauli
strings of every letter, on every site in turn, against the oracle.  Tolerances as in test_gpu_batch: 1e-10 of
<psi|psi> (FP64) and 1e-9 (mixed)."""
import numpy as np
import pytest

from oracle import chain_oracle as O
from qrochet import random as R
from qrochet import serve as S
from qrochet.batch import Batch

pytestmark = pytest.mark.gpu


def _request(chi, n, depth, seed):
    g = R.rng(seed)
    r = S.random_request(g, n_range=(n, n), depth_range=(depth, depth), chi_choices=(chi,), nobs=1)
    r.observables = [[]] + [[(s, "XYZ"[s % 3])] for s in range(1, n + 1)]
    r.observables += [[(s, "XYZ"[(s + k) % 3]) for k, s in enumerate(range(1, n + 1, 2))]]
    return r


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("chi,n,depth", [(1, 3, 2), (2, 2, 1), (3, 7, 5), (7, 9, 8), (9, 10, 8), (17, 11, 9),
                                         (31, 12, 10), (33, 13, 11), (63, 14, 12), (64, 14, 12)])
def test_odd_bonds_against_the_oracle(chi, n, depth, precision):
    tol = 1e-10 if precision == "fp64" else 1e-9
    r = _request(chi, n, depth, 100 * chi + n)
    with Batch(precision=precision) as b:
        rid = b.add(r)
        b.run()
        psi = O.from_reference_arrays(R.zero_product_arrays(n))
        for s, u in r.gates:
            O.evolve_2site_(psi, s - 1, u, threshold=r.threshold, maxdim=r.chi_max)
        ref = np.array([O.expect(psi, [O.ODense(R.PAULI[p], (O.OSite(s), O.OSite(s, True))) for s, p in o])
                        for o in r.observables])
        assert b.bond_dims(rid) == psi.bond_dims()
        for bond, lm in enumerate(psi.lam):
            got = b.lambda_on(rid, bond)
            assert (got is None) == (lm is None)
            if lm is not None:
                assert np.max(np.abs(got - lm)) <= tol * lm[0], bond
        assert np.max(np.abs(b.values(rid) - ref)) <= tol * max(abs(O.overlap(psi, psi)), 1e-300)
