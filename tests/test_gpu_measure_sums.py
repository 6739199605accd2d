"""Outcome probabilities and collapse over measured qubits in every position: lanes, thread bits, loop bits,
any order, duplicates, against numpy.  Tolerance: sums of 2^n squares in FP64 (FP32 squares: 2^-22 relative)."""
import numpy as np
import pytest

from tests.test_gaterun import random_state

pytestmark = pytest.mark.gpu


def outcome_of(n, qubits):
    i = np.arange(1 << n)
    return sum(((i >> q) & 1) << k for k, q in enumerate(qubits))


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("n,qubits", [(1, [0]), (2, [1]), (3, [2, 0]), (5, [4, 1, 2]), (6, [5]), (8, [0, 1, 2, 3, 4, 5, 6, 7]),
                                      (9, [8, 8, 2]), (12, [3]), (12, [11, 0, 6, 5]), (14, list(range(13, -1, -1))), (18, [17]),
                                      (19, [0, 9, 18, 4]), (20, list(range(2, 18)))])
def test_probabilities_and_collapse(qi, n, qubits, prec):
    prec = getattr(qi, prec)
    tol = 1e-12 if prec == qi.F64 else 1e-6
    psi = random_state(n, np.random.default_rng(n))
    with qi.DeviceState(n, prec) as s:
        s.upload(psi)
        o, probs = qi.measure(s, qubits, seed=5, return_probs=True)
        idx = outcome_of(n, qubits)
        want = np.bincount(idx, np.abs(psi) ** 2, minlength=1 << len(qubits))
        assert np.max(np.abs(probs - want)) <= tol
        assert o == int(np.searchsorted(np.cumsum(probs), qi.splitmix_uniform(5), side="right"))
        kept = np.where(idx == o, psi, 0)
        assert np.max(np.abs(s.download() - kept / np.linalg.norm(kept))) <= tol * 10
