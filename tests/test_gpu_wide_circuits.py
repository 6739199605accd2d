"""Small FP32 circuits and time steps that run in FP64 on a scratch copy: the rounded FP64 result, the state's own stream
or the caller's, errors that leave the state alone, and the norm that blocks would have given."""
import numpy as np
import pytest

from quant_iron_gb300 import F32, F64, FUSION_GREEDY, DeviceState, Plan, workloads
from quant_iron_gb300._abi import QuantIronError
from quant_iron_gb300.workloads import GateList
from tests.test_fp32_small_plans import ansatz, benchmark, evolution

pytestmark = pytest.mark.gpu


def psi_of(n, seed, norm=1.0):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return (norm * v / np.linalg.norm(v)).astype(np.complex64).astype(np.complex128)


@pytest.mark.parametrize("n,circuit", [(1, None), (2, None), (3, benchmark), (5, ansatz), (6, evolution), (9, evolution), (11, evolution)])
def test_circuits(qi, n, circuit):
    torch = pytest.importorskip("torch")
    if circuit is None:
        gl = GateList().add("H", [0]).add("RX", [n - 1], [], [0.3]).add("T", [0])
        gates = gl.add("PAULI_EVOLUTION", [], [], [1.0, 0.0, 0.2], xmask=1, zmask=1).array()
    else:
        gates = circuit(n, 4, n)
    for stream in (0, torch.cuda.Stream().cuda_stream):
        with DeviceState(n, F32) as a, DeviceState(n, F64) as b:
            a.set_stream(stream)
            a.upload(psi_of(n, n, 2.0))
            b.upload(psi_of(n, n, 2.0))
            qi.circuit_execute(a, gates, fusion=FUSION_GREEDY)
            qi.circuit_execute(b, gates)
            assert np.array_equal(a.download(), b.download().astype(np.complex64).astype(np.complex128))


def test_errors_leave_the_state_alone(qi):
    n = 4
    gates = GateList().add("H", [0]).add("PAULI_STRING", [], [], [1.0, 0.0], xmask=1, zmask=0).array()
    with DeviceState(n, F32) as a:
        a.upload(psi_of(n, 1))
        a.scale(0.0)
        with pytest.raises(QuantIronError) as e:   # normalises a state of zeros
            qi.circuit_execute(a, gates, fusion=FUSION_GREEDY)
        assert e.value.variant == "ZeroNorm" and not np.any(a.download())
        a.upload(psi_of(n, 1))
        with pytest.raises(QuantIronError):
            qi.circuit_execute(a, GateList().add("X", [0]).add("H", [7]).array(), fusion=FUSION_GREEDY)
        assert np.array_equal(a.download(), psi_of(n, 1))


def test_measurements_stay_in_fp32(qi):
    """Outcomes and collapsed states of a small circuit are the plan's (blocks)."""
    n = 5
    for seed in range(6):
        gates = GateList().add("H", [0]).add("RY", [1], [], [0.7]).add("CNOT", [2], [0]).measure([0, 1, 2], seed=seed).add("H", [3]).array()
        with DeviceState(n, F32) as a, DeviceState(n, F32) as b:
            a.upload(psi_of(n, 2))
            b.upload(psi_of(n, 2))
            qi.circuit_execute(a, gates, fusion=FUSION_GREEDY)
            Plan(n, F32, gates, fusion=FUSION_GREEDY).execute(b)
            assert np.max(np.abs(a.download() - b.download())) <= 16 * 2.0 ** -24


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("terms", ["xyz", "fields"])
def test_steps_of_twelve_qubits_on_a_state_of_another_norm(qi, terms, order):
    """Blocks on the tensor cores are followed by a renormalisation, diagonal runs are not: the same here."""
    n, dt, steps = 12, 0.05, 2
    t = workloads.lattice_xyz(3, 4, seed=2)
    if terms == "fields":
        t = t[t["xmask"] == 0]
    gl = GateList()
    for r in (t if order == 1 else np.concatenate([t, t[::-1]])):
        gl.add("PAULI_EVOLUTION", [], [], [r["re"], r["im"], dt / order], xmask=int(r["xmask"]), zmask=int(r["zmask"]))
    step = Plan(n, F32, gl.array(), fusion=FUSION_GREEDY, max_block_qubits=6)
    with DeviceState(n, F32) as a, DeviceState(n, F32) as b:
        a.upload(psi_of(n, 3, 2.0))
        b.upload(psi_of(n, 3, 2.0))
        qi.trotter_evolve(a, t, dt, steps, order)
        for _ in range(steps):
            step.execute(b)
        # blocks: a few 2^-24 per amplitude and step of 140 exponentials or fewer
        assert np.max(np.abs(a.download() - b.download())) <= 2.0 * 300 * 2.0 ** -24 * 2.0
        assert abs(a.norm_sqr() - b.norm_sqr()) <= 1e-3
