"""A recycled handle whose buffer leaves the engine: what an earlier owner, or a reader of its buffer, still has in
flight is over before the buffer can be written on another stream.  (A state that was never touched has no work a
caller could wait for.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from quant_iron_gb300 import workloads  # noqa: E402

pytestmark = pytest.mark.gpu
N = 17   # 2 MiB FP64: small enough to be recycled


class Memory:
    def __init__(self, state):
        self.__cuda_array_interface__ = {"data": (state.device_ptr(), False), "shape": (1 << state.n, 2), "typestr": "<f8",
                                         "version": 2}


def busy(plan, state, times=60):
    for _ in range(times):
        plan.execute(state)


def overwrite(qi, how, state):
    """Fill a new state with 0.5 + 0.5 i on a stream of the caller's own."""
    st = torch.cuda.Stream()
    if how == "pointer":
        with torch.cuda.stream(st):
            torch.as_tensor(Memory(state), device="cuda").fill_(0.5)
    else:
        state.set_stream(st.cuda_stream)
        state.set_plus()
        state.scale((0.5 + 0.5j) * 2.0 ** (N / 2))
    st.synchronize()


@pytest.mark.parametrize("how", ["pointer", "stream"])
@pytest.mark.parametrize("pending", ["reader", "owner"])
def test_new_owner_on_another_stream(qi, pending, how):
    plan = qi.Plan(N, qi.F64, workloads.random_circuit(N, layers=10, seed=1))
    with qi.DeviceState(N, qi.F64) as b, qi.DeviceState(N, qi.F64) as want:
        for s in (b, want):
            s.set_plus()
            plan.execute(s)
            s.synchronize()
        qi.trim_cache()
        a = qi.DeviceState(N, qi.F64)
        a.set_minus()
        a.synchronize()
        want.set_minus()
        if pending == "reader":
            busy(plan, b)      # b's stream reaches the copy late
            b.copy_from(a)
        else:
            busy(plan, a)
        a.close()              # kept, with that in flight
        c = qi.DeviceState(N, qi.F64)
        overwrite(qi, how, c)
        if pending == "reader":
            assert np.array_equal(b.download(), want.download())
        got = c.download()
        assert np.allclose(got, 0.5 + 0.5j, rtol=0, atol=1e-12)
        c.close()
