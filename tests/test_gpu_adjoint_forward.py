"""The forward pass of a gradient: fused blocks where a gate of the circuit cannot join a gate run, and whatever the
caller chose."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from quant_iron_gb300.workloads import GateList

pytestmark = pytest.mark.gpu


def ansatz(n, matchgates, seed):
    rng = np.random.default_rng(seed)
    gl, theta = GateList(), []
    for layer in range(4):
        for q in range(n):
            theta.append(float(rng.uniform(-3.0, 3.0)))
            gl.add(("RY", "RZ")[layer % 2], [q], [], [theta[-1]], [len(theta) - 1])
        for q in range(layer % 2, n - 1, 2):
            if matchgates:
                theta.append(float(rng.uniform(-3.0, 3.0)))
                gl.add("MATCHGATE", [q], [], [theta[-1], 0.3, 0.4], [len(theta) - 1])
            else:
                gl.add("CNOT", [q + 1], [q])
    return gl.array(), np.array(theta)


def gradient(qi, s, gates, theta, terms, **opts):
    l0 = qi.launch_count()
    e, g = qi.adjoint_gradient(s, gates, theta, terms, **opts)
    return e, g, qi.launch_count() - l0


@pytest.mark.parametrize("n", [12, 14, 16])
def test_matchgates_keep_fused_blocks(qi, n):
    """FP32: as many launches, and the same values, as with the default block size (5) named."""
    gates, theta = ansatz(n, True, n)
    terms = workloads.heisenberg_open_chain(n, seed=n)
    with qi.DeviceState(n, qi.F32) as s:
        s.set_zero()
        gradient(qi, s, gates, theta, terms)
        e, g, launches = gradient(qi, s, gates, theta, terms)
        e5, g5, launches5 = gradient(qi, s, gates, theta, terms, max_block_qubits=5)
        assert launches == launches5 and e == e5 and np.array_equal(g, g5)


@pytest.mark.parametrize("opts", [{"use_tensor_cores": 1}, {"use_tensor_cores": 2}, {"fusion": "learned"}])
@pytest.mark.parametrize("n", [13, 16])
def test_callers_options_hold(qi, n, opts):
    """A caller's choice of tensor cores, CUDA cores or learned partitions is what the forward pass runs."""
    opts = {k: qi.FUSION_LEARNED if v == "learned" else v for k, v in opts.items()}
    gates, theta = ansatz(n, False, n)
    terms = workloads.heisenberg_open_chain(n, seed=n)
    with qi.DeviceState(n, qi.F32) as s:
        s.set_zero()
        e, _, _ = gradient(qi, s, gates, theta, terms, **opts)
        e5, _, _ = gradient(qi, s, gates, theta, terms, max_block_qubits=5, **opts)
        assert e == e5
