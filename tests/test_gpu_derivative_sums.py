"""FP32 derivative terms: a thread's products are summed in FP32, threads are not.

RY(0) on a state of positive amplitudes and H = Z of the same qubit: no gate rounds anything, and all products of the
term have one sign.  A thread sums two chains of 8 products: half a unit in the last place at the size of each
partial sum is 0.5 u of a thread's sum (u = 2^-24), 0.03 u of the sum of 256 threads or more.  The root mean
square over qubits and seeds has to be within 0.15 u (FP32 sums over the block would leave 0.7 u)."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from quant_iron_gb300.workloads import GateList

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 14])
def test_terms_of_one_sign(qi, n):
    rel = []
    for seed in range(3):
        psi = np.random.default_rng(n + seed).uniform(0.5, 1.5, size=1 << n)
        psi = (psi / np.linalg.norm(psi)).astype(np.float32).astype(np.float64)
        with qi.DeviceState(n, qi.F32) as s:
            s.upload(psi)
            for q in range(n):
                gates = GateList().add("RY", [q], [], [0.0], [0]).array()
                terms = workloads.terms_array([workloads.term(1.0, [(q, "Z")])])
                _, g = qi.adjoint_gradient(s, gates, np.zeros(1), terms)
                v = psi.reshape(-1, 2, 1 << q)
                rel.append(g[0] / (-2.0 * float(np.sum(v[:, 0] * v[:, 1]))) - 1.0)
    assert np.sqrt(np.mean(np.square(rel))) <= 0.15 * 2.0 ** -24
