"""FP32 gradients of Hamiltonians of any size: coefficients times a power of two give energy and gradient times it."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from quant_iron_gb300.workloads import GateList

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angle", [np.pi / 2, 1.2])   # where a rotation's scale is smallest, and a generic one
@pytest.mark.parametrize("n", [5, 13])
def test_large_coefficients(qi, n, angle):
    gl, theta = GateList(), []
    for layer in range(60):
        for q in range(4):
            theta.append(angle + 1e-3 * q)
            gl.add("RX" if layer % 2 else "RY", [q], [], [theta[-1]], [len(theta) - 1])
    gates, theta = gl.array(), np.array(theta)
    terms = workloads.terms_array([workloads.term(1.0, [(0, "Z")]), workloads.term(0.75, [(1, "X"), (2, "X")])])
    with qi.DeviceState(n, qi.F32) as s:
        s.set_zero()
        e, g = qi.adjoint_gradient(s, gates, theta, terms)
        assert np.linalg.norm(g) > 1e-3
        for power in (10, 20, 40, 60, 80, 100):
            big = terms.copy()
            big["re"] *= 2.0 ** power
            e2, g2 = qi.adjoint_gradient(s, gates, theta, big)
            assert e2 == e * 2.0 ** power and np.array_equal(g2, g * 2.0 ** power), power
