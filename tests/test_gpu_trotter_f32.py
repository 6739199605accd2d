"""FP32 time steps are as exact as steps of fused blocks (each composed in FP64, rounded once): states of fewer than 12
qubits evolve in FP64, gate runs take over from blocks only from 13 qubits and three passes over the terms on."""
import numpy as np
import pytest

from quant_iron_gb300 import F32, F64, FUSION_GREEDY, DeviceState, Plan, workloads
from quant_iron_gb300.workloads import GateList

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [workloads.lattice_xyz, workloads.lattice_tfim])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("steps", [1, 3, 8])
@pytest.mark.parametrize("rows,cols", [(1, 3), (2, 2), (2, 3), (3, 3), (1, 11), (3, 4), (1, 13), (3, 5)])
def test_error_is_no_larger_than_blocks(qi, rows, cols, steps, order, model):
    """Root mean square of the error against FP64 over 8 basis states and Hamiltonians, with 20 % for the scatter of
    two such means (the errors of one small state are few numbers)."""
    n, dt, err, block_err = rows * cols, 0.05, [], []
    for seed in range(8):
        terms = model(rows, cols, seed=seed)
        seq = list(terms) if order == 1 else list(terms) + list(terms)[::-1]
        gl = GateList()
        for t in seq:
            gl.add("PAULI_EVOLUTION", [], [], [t["re"], t["im"], dt / order], xmask=int(t["xmask"]), zmask=int(t["zmask"]))
        step = Plan(n, F32, gl.array(), fusion=FUSION_GREEDY, max_block_qubits=6)
        basis = int(np.random.default_rng(seed).integers(0, 1 << n))
        with DeviceState(n, F32) as a, DeviceState(n, F32) as b, DeviceState(n, F64) as c:
            for s in (a, b, c):
                s.set_basis(basis)
            qi.trotter_evolve(a, terms, dt, steps, order)
            qi.trotter_evolve(c, terms, dt, steps, order)
            for _ in range(steps):
                step.execute(b)
            want = c.download()
            err.append(np.linalg.norm(a.download() - want))
            block_err.append(np.linalg.norm(b.download() - want))
    assert np.sqrt(np.mean(np.square(err))) <= 1.2 * np.sqrt(np.mean(np.square(block_err)))


@pytest.mark.parametrize("n", [2, 6, 11])
def test_small_states_are_the_rounded_fp64_evolution(qi, n):
    """Amplitudes, and observables on the way; a caller's stream and a state that was not normalised."""
    terms = workloads.heisenberg_open_chain(n, seed=n)
    rng = np.random.default_rng(n)
    psi = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)).astype(np.complex64).astype(np.complex128)
    torch = pytest.importorskip("torch")
    with DeviceState(n, F32) as a, DeviceState(n, F64) as b:
        a.upload(psi)
        b.upload(psi)
        a.synchronize()
        a.set_stream(torch.cuda.Stream().cuda_stream)
        ea = qi.trotter_evolve(a, terms, 0.05, 6, 2, observable=terms, observe_every=2)
        eb = qi.trotter_evolve(b, terms, 0.05, 6, 2, observable=terms, observe_every=2)
        assert np.array_equal(a.download(), b.download().astype(np.complex64).astype(np.complex128))
        assert np.array_equal(np.asarray(ea), np.asarray(eb))
