"""Calls that read another state, inside a relaxed capture of the written state's stream, the source on a stream of its
own: the source is waited for on the host, as outside a graph its stream is by an event."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from tests.test_gaterun import random_state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["copy_from", "axpy", "pauli_apply", "apply_gate_from"])
def test_reads_of_another_stream(qi, call):
    n = 10
    rng = np.random.default_rng(3)
    va, vb = random_state(n, rng), random_state(n, rng)
    term = workloads.terms_array([workloads.term(0.5, [(1, "X"), (4, "Y")])])[0]
    gate = workloads.GateList().add("H", [2]).array()[0]

    def run(dst, src):
        if call == "copy_from":
            dst.copy_from(src)
        elif call == "axpy":
            dst.axpy(0.5 - 0.25j, src)
        elif call == "pauli_apply":
            qi.pauli_apply(dst, src, term)
        else:
            dst.apply_gate_from(src, gate)

    st = torch.cuda.Stream()
    with qi.DeviceState(n, qi.F64) as a, qi.DeviceState(n, qi.F64) as b, qi.DeviceState(n, qi.F64) as want:
        a.upload(va)
        want.upload(vb)
        run(want, a)
        b.set_stream(st.cuda_stream)
        b.upload(vb)
        b.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st, capture_error_mode="relaxed"):
            run(b, a)
        with torch.cuda.stream(st):
            graph.replay()
        st.synchronize()
        assert np.array_equal(b.download(), want.download())
        assert np.array_equal(a.download(), va)   # the source's stream is not part of the graph
        b.upload(vb)
        run(b, a)                                  # and the same call outside
        assert np.array_equal(b.download(), want.download())
        del graph
