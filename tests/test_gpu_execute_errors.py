"""circuit_execute that fails on the way returns when nothing of it is running any more (its program lies in the
state's memory, which the next call may take on another stream)."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from quant_iron_gb300._abi import QuantIronError

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["F64", "F32"])
def test_a_failed_circuit_is_over(qi, prec):
    """A measurement (X basis) of a state of zeros fails; the change back of the basis is in flight then."""
    n = 24
    gl = workloads.GateList()
    for q in range(n):
        gl.add("H", [q]).add("T", [q])
    gl.measure(list(range(n)), basis=1)
    with qi.DeviceState(n, getattr(qi, prec)) as s:
        s.set_zero()
        s.scale(0.0)
        stream = torch.cuda.ExternalStream(s.stream())
        with pytest.raises(QuantIronError):
            qi.circuit_execute(s, gl.array())
        assert stream.query()
