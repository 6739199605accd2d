"""Adjoint gradients by tile passes over psi and lambda: every gate kind a pass takes, parameters of each kind,
controls and diagonal gates inside and outside the tile, tile edges, against the sweep of one pass per gate.

Tolerance: FP64 1e-10 of the gradient's norm (the per-gate sweep's own derivative matrices are good to 1e-12);
FP32 within 2e-5 (80 gates, each rounding both states by a few 2^-24)."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from quant_iron_gb300.workloads import GateList

pytestmark = pytest.mark.gpu


def parametric_circuit(n, gates, rng):
    gl, theta = GateList(), []
    fixed = ["H", "X", "Y", "Z", "S", "T", "SDAG", "TDAG", "CNOT", "SWAP", "P", "RX", "RY", "RZ"]
    for _ in range(gates):
        qs = [int(q) for q in rng.permutation(n)]
        if rng.random() < 0.5:
            theta.append(float(rng.uniform(-7.0, 7.0)))
            gl.add(("RX", "RY", "RZ", "P")[int(rng.integers(0, 4))], [qs[0]], [], [theta[-1]], [len(theta) - 1])
            continue
        k = fixed[int(rng.integers(0, len(fixed)))]
        a = [float(rng.uniform(-3.0, 3.0))] if k in ("P", "RX", "RY", "RZ") else []
        if k == "CNOT":
            gl.add(k, [qs[0]], [qs[1]])
        elif k == "SWAP":
            gl.add(k, qs[:2])
        else:
            gl.add(k, [qs[0]], qs[1:2] if rng.random() < 0.3 else [], a)
    theta.append(0.25)   # a parameter no gate uses
    return gl.array(), np.array(theta)


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 10, 11, 12, 13, 15, 18])
def test_tile_sweep_against_one_pass_per_gate(qi, n, prec):
    prec = getattr(qi, prec)
    rng = np.random.default_rng(n)
    gates, theta = parametric_circuit(n, 160, rng)
    terms = workloads.heisenberg_open_chain(n, seed=n)
    with qi.DeviceState(n, prec) as s, qi.DeviceState(n, qi.F64) as r:
        s.set_zero()
        r.set_zero()
        e, g = qi.adjoint_gradient(s, gates, theta, terms)
        e0, g0 = qi.adjoint_gradient(r, gates, theta, terms, fusion=qi.FUSION_NONE)
        tol = 1e-10 if prec == qi.F64 else 2e-5
        assert abs(e - e0) <= tol * len(terms)
        assert np.linalg.norm(g - g0) <= tol * max(1.0, np.linalg.norm(g0))
        assert g[-1] == 0.0
        e2, g2 = qi.adjoint_gradient(s, gates, theta, terms)   # the state is as it was
        assert e2 == e and np.array_equal(g, g2)


def test_special_angles(qi):
    """Angles where a rotation is the identity, a Pauli or swaps its larger entry."""
    n = 4
    gl, theta = GateList(), []
    for k, a in enumerate([0.0, np.pi, -np.pi, np.pi / 2, 2 * np.pi, 1e-9, 3 * np.pi / 2]):
        for name in ("RX", "RY", "RZ", "P"):
            gl.add("H", [k % n])
            theta.append(a)
            gl.add(name, [k % n], [], [a], [len(theta) - 1])
            gl.add("CNOT", [(k + 1) % n], [k % n])
    theta = np.array(theta)
    terms = workloads.xxz_periodic(n, seed=2)
    with qi.DeviceState(n, qi.F64) as s:
        s.set_plus()
        _, g = qi.adjoint_gradient(s, gl.array(), theta, terms)
        _, g0 = qi.adjoint_gradient(s, gl.array(), theta, terms, fusion=qi.FUSION_NONE)
        assert np.max(np.abs(g - g0)) <= 1e-10
