"""What a running request counts for in a server's budget: the gate step's peak, which the device memory taken by
one gate must not exceed; at most the budget, so that whatever is accepted also runs."""
import ctypes as C
import os
import subprocess
import sys

import pytest

from qrochet import _lib
from qrochet import serve as S

PKG = os.path.dirname(os.path.dirname(os.path.abspath(_lib.__file__)))

GATE = """
import sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
import qrochet as Q
from qrochet import random as R
chi = int(sys.argv[2])
g = R.rng(chi)
torch.zeros(1).cuda()
Q.zeros_chain(4)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
s = lambda *d: R.complex_gaussian(g, d) / np.sqrt(2 * chi)
psi = Q.MPS([s(2, chi), s(2, chi, chi), s(2, chi, chi), s(2, chi)])
psi.set_precision(sys.argv[3])
psi.set_lambda(1, 10.0 ** (-float(sys.argv[4]) * np.arange(chi) / chi))
Q.evolve_(psi, Q.gate_from_matrix(R.haar_unitary(g, 4), [2, 3]), threshold=1e-10, maxdim=chi)
torch.cuda.synchronize()
print(free - torch.cuda.mem_get_info()[0] - 16 * 4 * chi * (chi + 1))
"""


def admission(n, chi, budget):
    b = C.c_uint64()
    _lib.check(_lib.lib().qr_test_server_admission(n, chi, budget, C.byref(b)))
    return b.value


@pytest.mark.parametrize("n,chi", [(2, 1), (16, 64), (64, 1024)])
def test_accepted_requests_run(n, chi):
    f = S.footprint(n, chi)
    assert f <= admission(n, chi, 1 << 60)
    assert admission(n, chi, f) == f  # the smallest budget that accepts it: alone
    assert admission(n, chi, 1 << 60) <= f + 19 * 16 * (2 * chi) ** 2


@pytest.mark.gpu
@pytest.mark.parametrize("chi,precision,decades", [(300, "fp64", 0.5), (512, "mixed", 7.0), (512, "mixed", 0.5)])
def test_a_gate_stays_within_its_share(chi, precision, decades):
    out = subprocess.run([sys.executable, "-c", GATE, PKG, str(chi), precision, str(decades)], capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert int(out.stdout.split()[-1]) <= admission(2, chi, 1 << 60)
