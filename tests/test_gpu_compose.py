"""Blocks composed on the device (a circuit run in one call, a Trotter step, a gradient's forward sweep) against the
same blocks composed on the host (a plan).  Both compose in FP64, so their TF32 operands differ at most in the last
bit of the low part: 2^-22 of an amplitude a block."""
import numpy as np
import pytest

from tests.test_gaterun import mixed_circuit, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [3, 4, 5, 6])
@pytest.mark.parametrize("n", [11, 12, 13, 16, 21])
def test_one_call_against_a_plan(qi, n, k):
    rng = np.random.default_rng(100 * n + k)
    psi = random_state(n, rng)
    for gates in (mixed_circuit(n, 120, rng), mixed_circuit(n, 40, rng, exps=False)):
        plan = qi.Plan(n, qi.F32, gates, fusion=qi.FUSION_GREEDY, max_block_qubits=k)
        with qi.DeviceState(n, qi.F32) as a, qi.DeviceState(n, qi.F32) as b:
            a.upload(psi)
            b.upload(psi)
            for _ in range(2):
                plan.execute(a)
                qi.circuit_execute(b, gates, fusion=qi.FUSION_GREEDY, max_block_qubits=k)
            want, got = a.download(), b.download()
        assert np.max(np.abs(got - want)) <= 2 * len(gates) * 2.0 ** -22 * np.max(np.abs(want)), (n, k)
