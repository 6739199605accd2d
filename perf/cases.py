"""Timed workloads of the state-vector engine: what a user's program has it do, by size and option.

Every case goes through the public entry points of the package (the quant_iron mirror of the crate's
API, DeviceState, Plan, circuit_execute, trotter_evolve, sumop_*, adjoint_gradient, measure*).  Circuits
are the benchmark family (random single-qubit layers, CNOT brickwork, QFT), Hamiltonians the
package's Heisenberg / TFIM / XXZ generators; angles, circuits and initial states come from the seed.

exact() restates each workload in plain torch, complex128, with nothing from the package.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

qi = load_package()
from quant_iron_gb300 import quant_iron as api  # noqa: E402
from quant_iron_gb300 import workloads  # noqa: E402

PREC = {"f32": qi.F32, "f64": qi.F64}
REAL = {"f32": np.float32, "f64": np.float64}   # what is computed from a state is as exact as the state
FUSION = {"none": qi.FUSION_NONE, "greedy": qi.FUSION_GREEDY}
MEAN = 2.0                # of the amplitudes whose energy is taken, in standard deviations
EXACT_MAX_QUBITS = 23     # exact() of circuits, gradients and Trotter steps stays within seconds
ONE_QUBIT = ["H", "X", "Y", "Z", "S", "T", "RX", "RY", "RZ", "P"]


def listed():
    return [
        # a few gates on a small register through State's gate methods, read back after the last one:
        # notebooks, unit tests, the crate's own examples
        {"name": "methods_8q", "kind": "methods", "n": 8, "layers": 3},
        # Circuit.execute of a built circuit on a State, amplitudes read back (algorithm prototypes)
        {"name": "circuit_api_10q", "kind": "circuit_api", "n": 10, "layers": 10},
        # the plain method: 20 qubits, FP64 per gate, 40 layers + QFT, then <H> of the open Heisenberg chain
        {"name": "circuit_f64_20q", "kind": "circuit", "n": 20, "layers": 40, "prec": "f64", "fusion": "none"},
        # the same family at the size where the state no longer fits the L2
        {"name": "circuit_f64_25q", "kind": "circuit", "n": 25, "layers": 12, "prec": "f64", "fusion": "none"},
        # a compiled FP32 plan run again and again on a mid-size register (sampling, sweeps)
        {"name": "plan_f32_17q", "kind": "plan", "n": 17, "layers": 40, "prec": "f32", "fusion": "greedy"},
        # the headline workload: 30 qubits, 40 layers + QFT, fused complex FP32
        {"name": "plan_f32_30q", "kind": "plan", "n": 30, "layers": 40, "prec": "f32", "fusion": "greedy"},
        # time evolution of a random basis state on an open lattice, FP32
        {"name": "trotter_f32_4x6", "kind": "trotter", "rows": 4, "cols": 6, "model": "xyz", "prec": "f32", "steps": 5,
         "order": 1},
        # the same in FP64, second order, a register small enough for exact studies
        {"name": "trotter_f64_3x6", "kind": "trotter", "rows": 3, "cols": 6, "model": "tfim", "prec": "f64", "steps": 10,
         "order": 2},
        # energy and H|psi> (energy variance, Lanczos) of a large FP32 state
        {"name": "observable_f32_27q", "kind": "observable", "n": 27, "prec": "f32"},
        # one gradient of a small variational circuit, FP64: the inner loop of an optimiser
        {"name": "gradient_f64_12q", "kind": "gradient", "n": 12, "layers": 4, "prec": "f64"},
        # the gradient benchmark: 26 qubits, 12 layers, 624 parameters, FP32
        {"name": "gradient_f32_26q", "kind": "gradient", "n": 26, "layers": 12, "prec": "f32"},
        # repeated sampling of a prepared register and one collapsing measurement of some of its qubits
        {"name": "measure_f64_22q", "kind": "measure", "n": 22, "measured": 10, "shots": 4096, "prec": "f64"},
    ]


def draw(rng):
    kind = rng.choice(["methods", "circuit_api", "circuit", "circuit", "plan", "plan", "trotter", "trotter",
                       "observable", "gradient", "gradient", "measure"])
    prec = rng.choice(["f32", "f64"])
    if kind == "methods":
        return {"kind": kind, "n": rng.randint(3, 14), "layers": rng.randint(1, 5)}
    if kind == "circuit_api":
        return {"kind": kind, "n": rng.randint(4, 16), "layers": rng.randint(3, 20)}
    if kind == "circuit":
        # FP64 or FP32 per gate; deep circuits on few qubits, shallower ones on many
        n = rng.randint(8, 25)
        return {"kind": kind, "n": n, "layers": rng.randint(4, 40 if n <= 21 else 12), "prec": prec, "fusion": "none"}
    if kind == "plan":
        n = rng.randint(10, 29)
        return {"kind": kind, "n": n, "layers": rng.randint(10, 40), "prec": "f32", "fusion": "greedy"}
    if kind == "trotter":
        rows = rng.randint(2, 4)
        cols = rng.randint(3, 6)
        return {"kind": kind, "rows": rows, "cols": cols, "model": rng.choice(["xyz", "tfim"]), "prec": prec,
                "steps": rng.randint(1, 10 if rows * cols <= 20 else 4), "order": rng.choice([1, 2])}
    if kind == "observable":
        return {"kind": kind, "n": rng.randint(8, 27 if prec == "f32" else 24), "prec": prec}
    if kind == "gradient":
        return {"kind": kind, "n": rng.randint(6, 24 if prec == "f32" else 18), "layers": rng.randint(2, 12), "prec": prec}
    n = rng.randint(8, 26 if prec == "f32" else 24)
    return {"kind": "measure", "n": n, "measured": rng.randint(1, min(n, 16)), "shots": rng.randint(100, 10000),
            "prec": prec}


# --------------------------------------------------------------------------- inputs
def _rng(case, seed):
    return np.random.Generator(np.random.PCG64([int(seed) & 0xFFFFFFFF, 7]))


def _circuit(n, layers, rng):
    """(kind, targets, controls, params) of `layers` random layers with CNOT brickwork, then a QFT."""
    out = []
    for layer in range(layers):
        for q in range(n):
            name = ONE_QUBIT[int(rng.integers(0, 10))]
            par = [float(rng.uniform(0.0, 2.0 * math.pi))] if name in ("RX", "RY", "RZ", "P") else []
            out.append((name, [q], [], par))
        for a in range(layer % 2, n - 1, 2):
            out.append(("CNOT", [a + 1], [a], []))
    for i in range(n):
        out.append(("H", [i], [], []))
        for k in range(1, n - i):
            out.append(("P", [i], [i + k], [math.pi / 2 ** k]))
    for i in range(n // 2):
        out.append(("SWAP", [i, n - 1 - i], [], []))
    return out


def _rows(circuit):
    gl = workloads.GateList()
    for name, t, c, p in circuit:
        gl.add(name, t, c, p)
    return gl.array()


class _Memory:
    """A state's device buffer as torch sees it (zero copy); the tensor keeps it, and so the state, alive."""

    def __init__(self, state, shape, typestr):
        self.state, ptr = state, state.device_ptr()
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _view(state):
    """The amplitudes of a DeviceState as a (2^n, 2) torch tensor on the same memory."""
    return torch.as_tensor(_Memory(state, (1 << state.n, 2), "<f4" if state.precision == qi.F32 else "<f8"),
                           device="cuda")


def _fill(view, seed, mean):
    """A normalised random state from the seed: complex Gaussian amplitudes about a real `mean`
    (0: a state after a deep circuit; above 0: part of it is |+...+>, so that energies are of the
    order of the register)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    view.normal_(generator=g)
    view[:, 0].add_(mean)
    norm = float(torch.linalg.vector_norm(view, dtype=torch.float64))
    view.mul_(1.0 / norm)


def _state(n, prec, seed, mean=0.0):
    s = qi.DeviceState(n, PREC[prec])
    _fill(_view(s), seed, mean)
    torch.cuda.synchronize()
    return s


def _exact_state(n, prec, seed, mean=0.0):
    v = torch.empty((1 << n, 2), dtype=torch.float32 if prec == "f32" else torch.float64, device="cuda")
    _fill(v, seed, mean)
    return torch.view_as_complex(v.double().contiguous())


def _hamiltonian(case, rng):
    """Terms as [(coefficient, {qubit: 'X'|'Y'|'Z'})], in the order of the package's generators."""
    if case["kind"] in ("trotter",):
        rows, cols = case["rows"], case["cols"]
        n = rows * cols
        bonds = [(r * cols + c, r * cols + c + 1) for r in range(rows) for c in range(cols - 1)]
        bonds += [(r * cols + c, (r + 1) * cols + c) for r in range(rows - 1) for c in range(cols)]
        if case["model"] == "tfim":
            return ([(-float(rng.uniform(0.5, 1.5)), {a: "Z", b: "Z"}) for a, b in bonds]
                    + [(-1.0, {q: "X"}) for q in range(n)])
        j = (1.0, 0.8, 0.5)
    elif case["kind"] == "gradient":
        n = case["n"]
        bonds = [(i, (i + 1) % n) for i in range(n)]
        j = (1.0, 1.0, 0.5)
    else:
        n = case["n"]
        bonds = [(i, i + 1) for i in range(n - 1)]
        j = (1.0, 1.0, 1.0)
    out = [(c, {a: p, b: p}) for a, b in bonds for c, p in zip(j, "XYZ")]
    return out + [(float(rng.uniform(-1.0, 1.0)), {q: "Z"}) for q in range(n)]


def _term_rows(terms):
    return workloads.terms_array([workloads.term(c, list(ops.items())) for c, ops in terms])


def _method_calls(n, layers, rng):
    """Gate-method calls (name, arguments) of a small layered program."""
    out = [("h", (q,)) for q in range(n)]
    for _ in range(layers):
        for q in range(n):
            out.append((("rx", "ry", "rz", "p")[int(rng.integers(0, 4))], (q, float(rng.uniform(0.0, 2.0 * math.pi)))))
        out += [("cnot", (q, q + 1)) for q in range(n - 1)]
        out += [("t", (int(rng.integers(0, n)),)), ("s", (int(rng.integers(0, n)),))]
    return out


def _host_state(n, seed):
    r = np.random.Generator(np.random.PCG64([int(seed) & 0xFFFFFFFF, 11]))
    v = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    return v / np.linalg.norm(v)


def _ansatz(case, rng):
    """RY, RZ on every qubit and a CNOT ladder per layer; every angle a parameter."""
    n, layers = case["n"], case["layers"]
    theta = rng.uniform(-math.pi, math.pi, size=2 * layers * n)
    gl, plain = workloads.GateList(), []
    for layer in range(layers):
        for q in range(n):
            for k, name in enumerate(("RY", "RZ")):
                pid = 2 * (layer * n + q) + k
                gl.add(name, [q], [], [theta[pid]], [pid])
                plain.append((name, [q], [], [float(theta[pid])]))
        for q in range(n - 1):
            gl.add("CNOT", [q + 1], [q])
            plain.append(("CNOT", [q + 1], [q], []))
    return gl.array(), plain, theta


# --------------------------------------------------------------------------- the cases
def prepare(case, seed):
    kind, rng = case["kind"], _rng(case, seed)
    st = {"case": case}
    if kind == "methods":
        st["calls"] = _method_calls(case["n"], case["layers"], rng)
        st["psi"] = api.State.new(_host_state(case["n"], seed))
    elif kind == "circuit_api":
        rows = _rows(_circuit(case["n"], case["layers"], rng))
        st["circuit"] = api.Circuit([api.Gate(r) for r in rows], case["n"])
        st["psi"] = api.State.new(_host_state(case["n"], seed))
    elif kind in ("circuit", "plan"):
        n = case["n"]
        st["gates"] = _rows(_circuit(n, case["layers"], rng))
        st["psi"] = _state(n, case["prec"], seed)
        if kind == "circuit":
            st["terms"] = _term_rows(_hamiltonian(case, rng))
        else:
            st["plan"] = qi.Plan(n, PREC[case["prec"]], st["gates"], fusion=FUSION[case["fusion"]])
    elif kind == "trotter":
        st["terms"] = _term_rows(_hamiltonian(case, rng))
        n = case["rows"] * case["cols"]
        st["psi"] = qi.DeviceState(n, PREC[case["prec"]])
        st["psi"].set_basis(int(rng.integers(0, 1 << n)))
        st["psi"].synchronize()
    elif kind == "observable":
        st["terms"] = _term_rows(_hamiltonian(case, rng))
        st["psi"] = _state(case["n"], case["prec"], seed, MEAN)
        st["out"] = qi.DeviceState(case["n"], PREC[case["prec"]])
    elif kind == "gradient":
        st["gates"], _, st["theta"] = _ansatz(case, rng)
        st["terms"] = _term_rows(_hamiltonian(case, rng))
        st["psi"] = qi.DeviceState(case["n"], PREC[case["prec"]])
        st["psi"].set_zero()
        st["psi"].synchronize()
    else:
        st["psi"] = _state(case["n"], case["prec"], seed)
        st["work"] = qi.DeviceState(case["n"], PREC[case["prec"]])
        st["qubits"] = sorted(rng.choice(case["n"], size=case["measured"], replace=False).tolist())
        st["seed"] = int(seed) & 0xFFFFFF
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "methods":
        psi = st["psi"]
        for name, args in st["calls"]:
            psi = getattr(psi, name)(*args)
        return {"amplitudes": psi.state_vector}
    if kind == "circuit_api":
        return {"amplitudes": st["circuit"].execute(st["psi"]).state_vector}
    if kind == "circuit":
        qi.circuit_execute(st["psi"], st["gates"], fusion=FUSION[case["fusion"]])
        if case["prec"] == "f32":
            return {"amplitudes": _view(st["psi"])}
        energy = qi.sumop_expectation(st["psi"], st["terms"])
        return {"amplitudes": _view(st["psi"]), "energy": energy.real}
    if kind == "plan":
        st["plan"].execute(st["psi"])
        return {"amplitudes": _view(st["psi"])}
    if kind == "trotter":
        qi.trotter_evolve(st["psi"], st["terms"], 0.05, case["steps"], case["order"])
        return {"amplitudes": _view(st["psi"])}
    if kind == "observable":
        energy = qi.sumop_expectation(st["psi"], st["terms"])
        qi.sumop_apply(st["out"], st["psi"], st["terms"])
        return {"energy": REAL[case["prec"]](energy.real), "h_psi": _view(st["out"])}
    if kind == "gradient":
        energy, grads = qi.adjoint_gradient(st["psi"], st["gates"], st["theta"], st["terms"])
        return {"energy_gradient": np.append(grads, energy).astype(REAL[case["prec"]])}
    shots = qi.measure_n(st["psi"], case["shots"], st["qubits"], seed=st["seed"])
    st["work"].copy_from(st["psi"])
    outcome, probs = qi.measure(st["work"], st["qubits"], seed=st["seed"], return_probs=True)
    return {"shots": shots.view(np.int64), "outcome": outcome, "probabilities": probs.astype(REAL[case["prec"]]),
            "collapsed": _view(st["work"])}


def work(case):
    """One pass over the path's inputs and outputs; flops of the gates as 2x2 (or diagonal) updates."""
    kind = case["kind"]
    n = case["rows"] * case["cols"] if kind == "trotter" else case["n"]
    dim = float(1 << n)
    amp = 8 if case.get("prec") == "f32" else 16
    per = {"H": 4, "RX": 8, "RY": 6, "RZ": 6, "P": 3, "T": 3}   # flops per amplitude; the others move data

    def circuit_flops(layers):
        layer = n * sum(per.get(g, 0) for g in ONE_QUBIT) / len(ONE_QUBIT)
        return dim * (layers * layer + 4 * n + 1.5 * n * (n - 1) / 2)

    if kind == "methods":
        return {"bytes": 2 * amp * dim, "flops": dim * (4 * n + case["layers"] * (6 * n + 3))}
    if kind in ("circuit_api", "plan"):
        return {"bytes": 2 * amp * dim, "flops": circuit_flops(case["layers"])}
    if kind == "circuit":
        return {"bytes": 2 * amp * dim, "flops": circuit_flops(case["layers"]) + (dim * 6 * n if amp == 16 else 0)}
    terms = len(_hamiltonian(case, np.random.default_rng(0))) if kind != "measure" else 0
    if kind == "trotter":
        return {"bytes": 2 * amp * dim, "flops": dim * 4 * terms * case["steps"] * case["order"]}
    if kind == "observable":
        return {"bytes": 2 * amp * dim, "flops": dim * 8 * terms}
    if kind == "gradient":
        return {"bytes": 2 * amp * dim, "flops": dim * (2 * case["layers"] * n * (3 * 6 + 8) + 4 * terms)}
    return {"bytes": 3 * amp * dim, "flops": dim * 8}


# --------------------------------------------------------------------------- 64-bit values
def _mat(name, p):
    r = 1.0 / math.sqrt(2.0)
    if name == "H":
        return ((r, r), (r, -r))
    if name in ("X", "CNOT"):
        return ((0, 1), (1, 0))
    if name == "Y":
        return ((0, -1j), (1j, 0))
    if name in ("Z", "S", "T", "P"):
        a = {"Z": math.pi, "S": math.pi / 2, "T": math.pi / 4}.get(name) if not p else p[0]
        exact = {"Z": -1.0, "S": 1j}
        return ((1, 0), (0, exact.get(name, complex(math.cos(a), math.sin(a)))))
    c, s = math.cos(p[0] / 2), math.sin(p[0] / 2)
    if name == "RX":
        return ((c, -1j * s), (-1j * s, c))
    if name == "RY":
        return ((c, -s), (s, c))
    return ((complex(c, -s), 0), (0, complex(c, s)))   # RZ


def _pairs(psi, t, c=None):
    """Views of the amplitudes with bit t clear and set (and bit c set, when given)."""
    if c is None:
        v = psi.view(-1, 2, 1 << t)
        return v[:, 0], v[:, 1]
    hi, lo = max(t, c), min(t, c)
    v = psi.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    return (v[:, 0, :, 1], v[:, 1, :, 1]) if t == hi else (v[:, 1, :, 0], v[:, 1, :, 1])


def _gate(psi, gate):
    name, t, c, p = gate
    if name == "SWAP":
        hi, lo = max(t), min(t)
        v = psi.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
        a, b = v[:, 0, :, 1], v[:, 1, :, 0]
        keep = a.clone()
        a.copy_(b)
        b.copy_(keep)
        return
    m = _mat(name, p)
    a, b = _pairs(psi, t[0], c[0] if c else None)
    if m[0][1] == 0:
        if m[0][0] != 1:
            a.mul_(m[0][0])
        b.mul_(m[1][1])
        return
    keep = a.clone()
    a.mul_(m[0][0]).add_(b, alpha=m[0][1])
    b.mul_(m[1][1]).add_(keep, alpha=m[1][0])


def _pauli(psi, ops):
    out = psi
    for q, p in ops.items():
        v = out.view(-1, 2, 1 << q)
        if p == "Z":
            out = torch.stack((v[:, 0], -v[:, 1]), 1).reshape(-1)
        elif p == "X":
            out = torch.stack((v[:, 1], v[:, 0]), 1).reshape(-1)
        else:
            out = torch.stack((-1j * v[:, 1], 1j * v[:, 0]), 1).reshape(-1)
    return out


def _h_psi(psi, terms):
    out = torch.zeros_like(psi)
    for c, ops in terms:
        out.add_(_pauli(psi, ops), alpha=c)
    return out


def _real(psi):
    return torch.view_as_real(psi)


def exact(case, seed):
    kind, rng = case["kind"], _rng(case, seed)
    n = case["rows"] * case["cols"] if kind == "trotter" else case["n"]
    if kind == "methods":
        psi = torch.from_numpy(_host_state(n, seed)).cuda()
        for name, args in _method_calls(n, case["layers"], rng):
            if name == "cnot":
                _gate(psi, ("CNOT", [args[1]], [args[0]], []))
            else:
                _gate(psi, (name.upper(), [args[0]], [], list(args[1:])))
        return {"amplitudes": psi.cpu().numpy()}
    if kind == "circuit_api":
        psi = torch.from_numpy(_host_state(n, seed)).cuda()
        for g in _circuit(n, case["layers"], rng):
            _gate(psi, g)
        return {"amplitudes": psi.cpu().numpy()}
    if kind in ("circuit", "plan"):
        if n > EXACT_MAX_QUBITS + 2:
            return None
        psi = _exact_state(n, case["prec"], seed)
        for g in _circuit(n, case["layers"], rng):
            _gate(psi, g)
        if kind == "plan":
            return {"amplitudes": _real(psi)}
        if case["prec"] == "f32":
            return {"amplitudes": _real(psi)}
        energy = torch.vdot(psi, _h_psi(psi, _hamiltonian(case, rng)))
        return {"amplitudes": _real(psi), "energy": float(energy.real)}
    if kind == "trotter":
        if n > EXACT_MAX_QUBITS + 1:
            return None
        terms = _hamiltonian(case, rng)
        psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        psi[int(rng.integers(0, 1 << n))] = 1.0
        seq = [(0.05, t) for t in terms] if case["order"] == 1 else [(0.025, t) for t in terms + terms[::-1]]
        for _ in range(case["steps"]):
            for dt, (c, ops) in seq:
                psi = psi * math.cos(dt * c) + _pauli(psi, ops) * (-1j * math.sin(dt * c))
        return {"amplitudes": _real(psi)}
    if kind == "observable":
        terms = _hamiltonian(case, rng)
        psi = _exact_state(n, case["prec"], seed, MEAN)
        out = _h_psi(psi, terms)
        return {"energy": float(torch.vdot(psi, out).real), "h_psi": _real(out)}
    if kind == "gradient":
        if n > EXACT_MAX_QUBITS:
            return None
        _, circuit, theta = _ansatz(case, rng)
        psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        psi[0] = 1.0
        for g in circuit:
            _gate(psi, g)
        lam = _h_psi(psi, _hamiltonian(case, rng))
        energy = float(torch.vdot(psi, lam).real)
        grads, k = np.zeros(theta.size), theta.size
        for name, t, c, p in reversed(circuit):
            if p:   # d/dtheta exp(-i theta P / 2): 2 Re <lam| (-i/2) P |psi> = Im <lam| P |psi>
                k -= 1
                grads[k] = float(torch.vdot(lam, _pauli(psi, {t[0]: name[1]})).imag)
            back = (name, t, c, [-x for x in p])
            _gate(psi, back)
            _gate(lam, back)
        return {"energy_gradient": np.append(grads, energy)}
    psi = _exact_state(n, case["prec"], seed)
    qubits = sorted(rng.choice(n, size=case["measured"], replace=False).tolist())
    index = torch.zeros(1 << n, dtype=torch.int64, device="cuda")
    every = torch.arange(1 << n, dtype=torch.int64, device="cuda")
    for k, q in enumerate(qubits):
        index |= ((every >> q) & 1) << k
    probs = torch.zeros(1 << case["measured"], dtype=torch.float64, device="cuda")
    probs.index_add_(0, index, psi.abs().square())
    probs /= probs.sum()
    # the drawn outcomes are whole numbers of the engine's own seeded generator
    return {"shots": None, "outcome": None, "probabilities": probs.cpu().numpy(), "collapsed": None}
