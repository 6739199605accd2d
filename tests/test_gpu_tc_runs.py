"""Tensor-core blocks whose tiles are 1, 2, ..., 2^k runs of memory: the producer warp copies a run per
lane, 64 runs in two rounds.  Compared with numpy FP64 within 1e-6 per amplitude (22 significant bits of
the split products on amplitudes of about 2^-10, as for one block in general); 22 qubits are several
tiles per persistent block."""
import numpy as np
import pytest

from tests.test_gpu_tensorcore import apply_np, haar, rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [5, 6])
@pytest.mark.parametrize("n", [15, 22])
def test_tensor_core_blocks_by_run_count(qi, k, n):
    init = rand_state(n, 2)
    for nhigh in range(k + 1):
        targets = list(range(k - nhigh)) + list(range(n - nhigh, n))
        U = haar(k, 50 + nhigh)
        with qi.DeviceState(n, qi.F32) as st:
            st.upload(init)
            qi.apply_matrix(st, targets, U, use_tensor_cores=1)
            got = st.download()
        assert np.max(np.abs(got - apply_np(init, n, targets, U))) < 1e-6, targets


@pytest.mark.parametrize("n", [19, 21, 23])
def test_back_to_back_blocks(qi, n):
    """Each launch sets up while the one before ends: a plan's blocks back to back, on two states in turn
    without a wait between, against the same plan with a wait after every execution (bit for bit) and
    against FP64 gates.  Tolerance: 50 blocks of 2^-21 relative error on amplitudes of at most 2^-6."""
    from quant_iron_gb300 import workloads
    gates = workloads.random_circuit(n, layers=6, seed=n)
    plan = qi.Plan(n, qi.F32, gates, fusion=qi.FUSION_GREEDY, use_tensor_cores=1)
    exact = qi.Plan(n, qi.F64, gates, fusion=qi.FUSION_NONE)
    with qi.DeviceState(n, qi.F32) as a, qi.DeviceState(n, qi.F32) as b, qi.DeviceState(n, qi.F32) as c, \
            qi.DeviceState(n, qi.F64) as d:
        for s in (a, b, c, d):
            s.set_plus()
        for _ in range(3):
            plan.execute(a)
            plan.execute(b)
        for _ in range(3):
            plan.execute(c)
            c.synchronize()
            exact.execute(d)
        got, want = a.download(), d.download()
        assert np.array_equal(got, b.download()) and np.array_equal(got, c.download())
    assert np.max(np.abs(want)) < 2.0 ** -6
    assert np.max(np.abs(got - want)) < 50 * 2.0 ** -21 * 2.0 ** -6


@pytest.mark.parametrize("n, prec", [(12, "F64"), (16, "F32"), (21, "F32")])
def test_chained_launches_on_other_streams_and_in_graphs(qi, n, prec):
    """The default stream, a caller's stream and a replayed graph of a plan's execution (gate runs at 12 and
    16 qubits, tensor-core blocks at 21) give what the state's own stream gives, bit for bit."""
    torch = pytest.importorskip("torch")
    from quant_iron_gb300 import workloads
    gates = workloads.random_circuit(n, layers=5, seed=n)
    plan = qi.Plan(n, getattr(qi, prec), gates, fusion=qi.FUSION_GREEDY if prec == "F32" else qi.FUSION_NONE)
    with qi.DeviceState(n, getattr(qi, prec)) as own, qi.DeviceState(n, getattr(qi, prec)) as s:
        own.set_plus()
        for _ in range(4):
            plan.execute(own)
        want = own.download()
        st = torch.cuda.Stream()
        for stream in (0, st.cuda_stream):
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
