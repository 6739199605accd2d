"""FP32 gradients: the forward pass is no less exact than fused blocks (block size named), whatever the size and depth,
and treats a state of another norm as blocks do."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from quant_iron_gb300.workloads import GateList

pytestmark = pytest.mark.gpu


def ansatz(n, layers, rng):
    gl, theta = GateList(), rng.uniform(-np.pi, np.pi, size=2 * n * layers)
    k = 0
    for _ in range(layers):
        for q in range(n):
            for name in ("RY", "RZ"):
                gl.add(name, [q], [], [theta[k]], [k])
                k += 1
        for q in range(n - 1):
            gl.add("CNOT", [q + 1], [q])
    return gl.array(), theta


@pytest.mark.parametrize("layers", [2, 6, 12])
@pytest.mark.parametrize("n", [3, 4, 5, 7, 9, 11, 12, 14, 16, 18])
def test_error_is_no_larger_than_with_blocks(qi, n, layers):
    """Root mean square over 8 seeds of the gradient's error against FP64, relative to its norm, with 15 % for the
    scatter of two such means."""
    err = {0: [], 5: []}
    for seed in range(8):
        gates, theta = ansatz(n, layers, np.random.default_rng(100 * n + seed))
        terms = workloads.heisenberg_open_chain(n, seed=seed)
        with qi.DeviceState(n, qi.F32) as a, qi.DeviceState(n, qi.F64) as b:
            a.set_zero()
            b.set_zero()
            _, want = qi.adjoint_gradient(b, gates, theta, terms)
            for block in err:
                _, g = qi.adjoint_gradient(a, gates, theta, terms, max_block_qubits=block)
                err[block].append(np.linalg.norm(g - want) / np.linalg.norm(want))
    assert np.sqrt(np.mean(np.square(err[0]))) <= 1.15 * np.sqrt(np.mean(np.square(err[5])))


@pytest.mark.parametrize("layers", [2, 12])
@pytest.mark.parametrize("n", [8, 14])
def test_states_of_another_norm(qi, n, layers):
    """|psi_0| = 2, against the call with blocks: energies within FP32 rounding of up to 500 gates."""
    gates, theta = ansatz(n, layers, np.random.default_rng(n))
    terms = workloads.heisenberg_open_chain(n, seed=n)
    with qi.DeviceState(n, qi.F32) as s:
        s.set_zero()
        s.scale(2.0)
        e, g = qi.adjoint_gradient(s, gates, theta, terms)
        e5, g5 = qi.adjoint_gradient(s, gates, theta, terms, max_block_qubits=5)
        assert abs(e - e5) <= 500 * 2.0 ** -24 * 4.0 * len(terms)
        assert np.linalg.norm(g - g5) <= 500 * 2.0 ** -24 * 4.0 * len(terms)
