"""Operator.apply takes what gate_row takes: qubits from any iterable, and rows that a subclass builds itself."""
import numpy as np
import pytest

from quant_iron_gb300 import quant_iron as api

pytestmark = pytest.mark.gpu


def test_qubits_from_any_iterable():
    s = api.State.new_plus(3)
    want = api.CNOT().apply(s, [1], [0]).state_vector
    for targets, controls in ((iter([1]), iter([0])), (np.array([1]), np.array([0])), (range(1, 2), (0,)),
                              ((q for q in [1]), {0}), ([1.0], [0])):
        assert np.array_equal(api.CNOT().apply(s, targets, controls).state_vector, want)


def test_rows_of_a_subclass():
    class Half(api.RotateX):
        """RX by half the angle."""
        def gate_row(self, targets, controls):
            row = super().gate_row(targets, controls).copy()
            row["params"][0] = 0.5 * self.angle
            return row

    s = api.State.new_plus(2).p(0, 0.7)
    assert np.array_equal(Half(1.2).apply(s, [0]).state_vector, api.RotateX(0.6).apply(s, [0]).state_vector)
