"""Runs of per-gate operations on the GPU: tile edges, controls and diagonal qubits outside the tile, both
precisions, against the oracle, and against one kernel per gate at sizes of many tiles.

Tolerance: a gate's update rounds each amplitude by a few units in the last place of the state's norm (1), so G
gates stay within 8 G u in the largest amplitude, u = 2^-53 or 2^-24."""
import numpy as np
import pytest

from tests.test_gaterun import mixed_circuit, random_state

pytestmark = pytest.mark.gpu


def unit(qi, prec):
    return 2.0 ** -53 if prec == qi.F64 else 2.0 ** -24


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 9, 10, 11, 12, 13, 14, 15])
def test_mixed_circuits_against_the_oracle(qi, orc, n, prec):
    prec = getattr(qi, prec)
    rng = np.random.default_rng(1000 + n)
    gates = mixed_circuit(n, 150, rng)
    init = random_state(n, rng)
    want = orc.execute(init, n, gates)
    with qi.DeviceState(n, prec) as s:
        s.upload(init)
        qi.circuit_execute(s, gates)
        assert np.max(np.abs(s.download() - want)) <= 8 * len(gates) * unit(qi, prec)


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("n", [20, 22, 23])
def test_many_tiles_against_one_kernel_per_gate(qi, n, prec):
    prec = getattr(qi, prec)
    gates = mixed_circuit(n, 120, np.random.default_rng(n))
    with qi.DeviceState(n, prec) as a, qi.DeviceState(n, qi.F64) as b:
        for s in (a, b):
            s.set_plus()
        plan = qi.Plan(n, prec, gates)
        passes, _, single = plan.run_info()   # FP32 passes take X strings of up to two qubits
        assert passes > 0 and (prec == qi.F32 or single == 0)
        plan.execute(a)
        for g in gates:
            b.apply_gate(g)
        assert a.compare(b)["max_abs_err"] <= 8 * len(gates) * unit(qi, prec)
