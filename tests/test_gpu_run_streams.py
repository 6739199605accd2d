"""Gate runs and blocks on the legacy default stream, the per-thread default stream and a caller's stream, and FP32 gate
runs in a replayed graph: what the state's own stream gives, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from quant_iron_gb300 import workloads  # noqa: E402

pytestmark = pytest.mark.gpu
LEGACY, PER_THREAD = 1, 2   # cudaStreamLegacy, cudaStreamPerThread


@pytest.mark.parametrize("n,prec,fusion", [(12, "F32", "GREEDY"), (14, "F32", "NONE"), (16, "F32", "GREEDY"), (14, "F64", "NONE")])
def test_streams_and_graphs(qi, n, prec, fusion):
    prec = getattr(qi, prec)
    gates = workloads.random_circuit(n, layers=6, seed=n)
    plan = qi.Plan(n, prec, gates, fusion=getattr(qi, "FUSION_" + fusion))
    with qi.DeviceState(n, prec) as own, qi.DeviceState(n, prec) as s:
        own.set_plus()
        for _ in range(4):
            plan.execute(own)
        want = own.download()
        st = torch.cuda.Stream()
        for stream in (LEGACY, PER_THREAD, st.cuda_stream):
            s.set_stream(stream)
            s.set_plus()
            for _ in range(4):
                plan.execute(s)
            assert np.array_equal(s.download(), want), stream
        s.set_plus()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            plan.execute(s)
            plan.execute(s)
        with torch.cuda.stream(st):
            graph.replay()
            graph.replay()
        st.synchronize()
        assert np.array_equal(s.download(), want)
        del graph


def test_one_call_circuits_on_the_default_streams(qi):
    n = 14
    gates = workloads.random_circuit(n, layers=6, seed=3)
    with qi.DeviceState(n, qi.F32) as own, qi.DeviceState(n, qi.F32) as s:
        own.set_plus()
        qi.circuit_execute(own, gates, fusion=qi.FUSION_GREEDY)
        for stream in (LEGACY, PER_THREAD):
            s.set_stream(stream)
            s.set_plus()
            qi.circuit_execute(s, gates, fusion=qi.FUSION_GREEDY)
            assert np.array_equal(s.download(), own.download())
