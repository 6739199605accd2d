"""Circuit.gate_array: an array of the caller's own, as writable as one built row by row."""
import numpy as np

from quant_iron_gb300 import quant_iron as api
from quant_iron_gb300.workloads import GateList


def test_rows_can_be_assigned():
    rows = GateList().add("H", [0]).add("RX", [1], [], [0.25]).add("CNOT", [1], [0]).array()
    circuit = api.Circuit([api.Gate(r) for r in rows], 2)
    a = circuit.gate_array()
    assert a.flags.writeable
    a["params"][1, 0] = 0.5
    assert a["params"][1, 0] == 0.5 and np.array_equal(circuit.gate_array(), rows)
