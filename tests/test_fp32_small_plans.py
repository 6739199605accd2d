"""FP32 circuits execute as gate runs only where a run's rounding of every gate is no worse than fused blocks' (composed
in FP64, rounded once per block of up to six qubits): not below 7 qubits, where a block holds the state or nearly, and
not with Pauli exponentials (near the identity, so a block hardly rounds) below 13."""
import numpy as np
import pytest

from quant_iron_gb300 import F32, F64, FUSION_GREEDY, DeviceState, Plan, workloads
from quant_iron_gb300.workloads import GateList


def benchmark(n, layers, seed):
    return workloads.random_circuit(n, layers=layers, seed=seed)


def ansatz(n, layers, seed):
    rng, gl = np.random.default_rng(seed), GateList()
    for _ in range(layers):
        for q in range(n):
            gl.add("RY", [q], [], [rng.uniform(-3, 3)]).add("RZ", [q], [], [rng.uniform(-3, 3)])
        for q in range(n - 1):
            gl.add("CNOT", [q + 1], [q])
    return gl.array()


def evolution(n, layers, seed):
    gl = GateList()
    for _ in range(layers):
        for t in workloads.heisenberg_open_chain(n, seed=seed):
            gl.add("PAULI_EVOLUTION", [], [], [t["re"], t["im"], 0.05], xmask=int(t["xmask"]), zmask=int(t["zmask"]))
    return gl.array()


@pytest.mark.parametrize("n", [4, 10, 11, 12, 13])
def test_which_plans_are_gate_runs(n):
    for circuit, runs in ((benchmark, 10 <= n <= 12), (ansatz, 10 <= n <= 12), (evolution, False)):
        plan = Plan(n, F32, circuit(n, 3, n), fusion=FUSION_GREEDY)
        assert (plan.run_info() != (0, 0, 0)) == runs


@pytest.mark.gpu
@pytest.mark.parametrize("circuit", [benchmark, ansatz, evolution])
@pytest.mark.parametrize("layers", [1, 10, 30])
@pytest.mark.parametrize("n", [4, 5, 6, 7, 9, 10, 12, 13])
def test_error_is_no_larger_than_blocks(qi, n, layers, circuit):
    """One-call circuits against the same with blocks (block size named), both against FP64: the root mean square
    of the error over 8 seeds, with 10 % for the scatter of two such means."""
    err = {0: [], 6: []}
    for seed in range(8):
        gates = circuit(n, layers, seed)
        rng = np.random.default_rng(seed)
        psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        psi = (psi / np.linalg.norm(psi)).astype(np.complex64).astype(np.complex128)
        with DeviceState(n, F32) as a, DeviceState(n, F64) as b:
            b.upload(psi)
            qi.circuit_execute(b, gates)
            want = b.download()
            for block in err:
                a.upload(psi)
                qi.circuit_execute(a, gates, fusion=FUSION_GREEDY, max_block_qubits=block)
                err[block].append(np.linalg.norm(a.download() - want))
    assert np.sqrt(np.mean(np.square(err[0]))) <= 1.1 * np.sqrt(np.mean(np.square(err[6])))
