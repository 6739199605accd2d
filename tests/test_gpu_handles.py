"""Gates from one state into another in one launch, and the cache of destroyed small handles: results are the copy's
bit for bit, readers of a buffer are waited for before its next owner writes, threads do not share."""
import threading

import numpy as np
import pytest

from quant_iron_gb300 import quant_iron as api
from quant_iron_gb300._abi import QuantIronError
from tests.test_gaterun import mixed_circuit, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("n", [1, 2, 3, 6, 11])
def test_gate_into_another_state_is_the_gate_on_a_copy(qi, n, prec):
    prec = getattr(qi, prec)
    rng = np.random.default_rng(n)
    psi = random_state(n, rng)
    gates = mixed_circuit(n, 60, rng) if n >= 3 else None
    if gates is None:
        from quant_iron_gb300.workloads import GateList
        gl = GateList()
        for k in ("H", "X", "Y", "Z", "S", "T", "IDENTITY"):
            gl.add(k, [n - 1])
        gates = gl.add("RX", [0], [], [0.4]).add("P", [0], list(range(1, n)), [1.1]).array()
    with qi.DeviceState(n, prec) as a, qi.DeviceState(n, prec) as b, qi.DeviceState(n, prec) as c:
        a.upload(psi)
        before = a.download()
        for g in gates:
            b.apply_gate_from(a, g)
            c.copy_from(a)
            c.apply_gate(g)
            assert np.array_equal(b.download(), c.download())
            assert np.array_equal(a.download(), before)


def test_errors_are_those_of_the_gate(qi):
    s = api.State.new_zero(3)
    for call in (lambda: s.h(3), lambda: s.cnot(1, 1), lambda: s.toffoli(0, 0, 5), lambda: s.swap(0, 0)):
        with pytest.raises(QuantIronError):
            call()
    with qi.DeviceState(3, qi.F64) as a, qi.DeviceState(4, qi.F64) as b, pytest.raises(QuantIronError):
        a.apply_gate_from(b, api.Hadamard().gate_row([0], []))


def chain(n, seed, rounds):
    """Gates, sums and Pauli strings on states that are dropped while their readers may still run."""
    rng = np.random.default_rng(seed)
    st = api.State.new(random_state(n, rng))
    for k in range(rounds):
        q = int(rng.integers(0, n - 1))
        st = st.h(q).rx(q, 0.1 * k).cnot(q, q + 1).t(q + 1)
        st = st * 0.5 + api.PauliString(0.5, {q: api.Pauli.Z}).apply(st)
        st = st.normalise()
    return st.state_vector


def test_reused_handles_give_the_same_states(qi):
    want = {(n, s): chain(n, s, 12) for n in (4, 9, 15) for s in range(3)}
    qi.trim_cache()
    got, errors = {}, []

    def work(n, s):
        try:
            got[n, s] = chain(n, s, 12)
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=k) for k in want]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k in want:
        assert np.array_equal(got[k], want[k])


def test_cache_is_bounded_and_leaves_exposed_buffers_alone(qi):
    import torch
    states = [qi.DeviceState(18, qi.F64) for _ in range(100)]   # what the driver keeps for 100 streams
    del states
    qi.trim_cache()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        states = [qi.DeviceState(18, qi.F64) for _ in range(100)]   # 4 MiB each
        del states
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 100 << 20
    qi.trim_cache()
    assert free0 - torch.cuda.mem_get_info()[0] <= 16 << 20
    a = qi.DeviceState(10, qi.F64)
    ptr = a.device_ptr()
    a.close()
    others = [qi.DeviceState(10, qi.F32) for _ in range(4)]
    assert ptr and others   # the exposed buffer was freed, not handed on by the cache
