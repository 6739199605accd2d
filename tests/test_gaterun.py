"""Runs of per-gate operations (several to a pass): schedule and programs against the oracle, on the CPU.

The passes of an FP64 plan are replayed on the host (qi_plan_run_replay) and compared with the oracle's gate by
gate result: every gate kind the passes take, controls and diagonal qubits inside and outside the tile, tiles
smaller than the state, more gates than one pass's program holds.

Tolerance: a gate's update rounds each amplitude by a few units of 2^-53 of the state's norm (1), so G gates stay
within 8 G 2^-53 in the largest amplitude; the scaled forms keep every intermediate entry at most 1.
"""
import numpy as np
import pytest

from quant_iron_gb300 import F64, FUSION_NONE, FUSION_PAULI_GROUPS, Plan, workloads
from quant_iron_gb300.workloads import GateList

EPS = 2.0 ** -53


def random_state(n, rng):
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return v / np.linalg.norm(v)


def unitary(rng):
    q, _ = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))
    return q


def mixed_circuit(n, gates, rng, exps=True):
    """Gates of every kind the passes take, with up to three controls and Pauli strings of any Z weight."""
    gl = GateList()
    kinds = ["H", "X", "Y", "Z", "S", "T", "SDAG", "TDAG", "P", "RX", "RY", "RZ", "U2", "RYPHASE", "RYPHASE_DAG", "CNOT",
             "SWAP", "TOFFOLI", "IDENTITY"] + (["EXP", "EXPZ"] if exps else [])
    for _ in range(gates):
        k = kinds[int(rng.integers(0, len(kinds)))]
        qs = [int(q) for q in rng.permutation(n)]
        nc = int(rng.integers(0, min(3, n - 1) + 1)) if rng.random() < 0.4 else 0
        a = [float(x) for x in rng.uniform(-7.0, 7.0, size=3)]
        if k in ("EXP", "EXPZ"):
            wx = 0 if k == "EXPZ" else int(rng.integers(1, min(3, n) + 1))
            wz = int(rng.integers(1, n + 1))
            x = sum(1 << q for q in qs[:wx])
            z = sum(1 << int(q) for q in rng.permutation(n)[:wz])
            gl.add("PAULI_EVOLUTION", [], [], [a[0], 0.0, 0.3], xmask=x, zmask=z)
        elif k == "CNOT":
            gl.add(k, [qs[0]], [qs[1]])
        elif k == "TOFFOLI":
            if n >= 3:
                gl.add(k, [qs[0]], qs[1:3])
        elif k == "SWAP":
            gl.add(k, qs[:2], qs[2:2 + min(nc, n - 2)])
        elif k == "U2":
            u = unitary(rng)
            gl.add(k, [qs[0]], qs[1:1 + nc], [f(u[i, j]) for i in (0, 1) for j in (0, 1) for f in (np.real, np.imag)])
        else:
            par = {"P": 1, "RX": 1, "RY": 1, "RZ": 1, "RYPHASE": 2, "RYPHASE_DAG": 2}.get(k, 0)
            gl.add(k, [qs[0]], qs[1:1 + nc], a[:par])
    return gl.array()


@pytest.mark.parametrize("n", [3, 4, 5, 8, 9, 10, 11, 12, 13, 14])
@pytest.mark.parametrize("fusion", [FUSION_NONE, FUSION_PAULI_GROUPS])
def test_replay_mixed_circuits(orc, n, fusion):
    rng = np.random.default_rng(100 * n + fusion)
    gates = mixed_circuit(n, 150, rng)
    init = random_state(n, rng)
    plan = Plan(n, F64, gates, fusion=fusion)
    passes, phases, single = plan.run_info()
    assert single == 0 and 0 < passes < len(gates)
    want = orc.execute(init, n, gates)
    assert np.max(np.abs(plan.run_replay(init) - want)) <= 8 * len(gates) * EPS


@pytest.mark.parametrize("n,layers", [(10, 40), (13, 12), (16, 4)])
def test_replay_benchmark_family(orc, n, layers):
    gates = workloads.random_circuit(n, layers=layers, seed=n)
    plan = Plan(n, F64, gates)
    init = workloads.plus_state(n)
    want = orc.execute(init, n, gates)
    assert np.max(np.abs(plan.run_replay(init) - want)) <= 8 * len(gates) * EPS


def test_scales_of_a_long_run_stay_in_range(orc):
    """3000 Hadamards leave out 2^-1500: the product is applied before the amplitudes overflow."""
    n = 5
    gl = GateList()
    for k in range(3000):
        gl.add("H", [(k * 2) % n])
        gl.add("RY", [(k * 3) % n], [], [0.7 + 1e-3 * k])
    gates = gl.array()
    init = random_state(n, np.random.default_rng(5))
    got = Plan(n, F64, gates).run_replay(init)
    assert np.max(np.abs(got - orc.execute(init, n, gates))) <= 8 * len(gates) * EPS


def test_runs_end_at_other_operations():
    """Matchgates, Pauli strings, wide X strings and measurements keep their own launches."""
    n = 6
    gl = GateList().add("H", [0]).add("T", [1]).add("MATCHGATE", [2], [], [0.3, 0.4, 0.5]).add("H", [3])
    gl.add("PAULI_STRING", [], [], [1.0, 0.0], xmask=3, zmask=1).add("X", [1]).add("Y", [2])
    gl.add("PAULI_EVOLUTION", [], [], [0.3, 0.0, 0.2], xmask=15, zmask=1)
    gl.measure([0, 1])
    plan = Plan(n, F64, gl.array())
    assert plan.run_info()[0::2] == (2, 5)
    with pytest.raises(Exception):
        plan.run_replay(random_state(n, np.random.default_rng(0)))


@pytest.mark.parametrize("rows,cols,terms", [(2, 3, workloads.lattice_tfim), (3, 4, workloads.lattice_xyz)])
def test_equal_exponentials_join(orc, rows, cols, terms):
    """Two second-order steps: terms that meet in the middle and at the boundary join, the rest keep their order."""
    n, t, dt = rows * cols, terms(rows, cols, seed=3), 0.1
    order = list(range(len(t))) + list(range(len(t)))[::-1]
    gl = GateList()
    for k in order + order:
        gl.add("PAULI_EVOLUTION", [], [], [t[k]["re"], t[k]["im"], dt / 2], xmask=int(t[k]["xmask"]), zmask=int(t[k]["zmask"]))
    gates = gl.array()
    init = random_state(n, np.random.default_rng(n))
    plan = Plan(n, F64, gates, fusion=FUSION_PAULI_GROUPS)
    assert np.max(np.abs(plan.run_replay(init) - orc.execute(init, n, gates))) <= 8 * len(gates) * EPS
