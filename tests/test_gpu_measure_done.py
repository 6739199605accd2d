"""measure returns when the state has collapsed: a reader of its buffer on any other stream sees the state that
download gives."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class Memory:
    def __init__(self, state):
        self.__cuda_array_interface__ = {"data": (state.device_ptr(), False), "shape": (1 << state.n, 2),
                                         "typestr": "<f4" if state.precision else "<f8", "version": 2}


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("basis", ["Computational", "X"])
def test_collapsed_on_return(qi, basis, prec):
    n = 24
    with qi.DeviceState(n, getattr(qi, prec)) as s:
        view = torch.as_tensor(Memory(s), device="cuda")
        stream = torch.cuda.ExternalStream(s.stream())
        for seed in range(3):
            s.set_plus()
            s.synchronize()
            qi.measure(s, [3, 7, 20], basis=basis, seed=seed)
            assert stream.query()
            seen = view.clone()
            torch.cuda.synchronize()
            assert np.array_equal(seen.double().cpu().numpy().reshape(-1).view(np.complex128), s.download())
