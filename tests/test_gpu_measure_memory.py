"""Measuring many qubits takes its sums' memory for the call alone, not for the life of the state."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,measured", [(24, 24), (24, 21), (22, 10)])
def test_sums_are_given_back(qi, n, measured):
    with qi.DeviceState(n, qi.F32) as s:
        s.set_plus()
        qi.measure_n(s, 10, [0])   # the small workspace
        s.synchronize()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        qi.measure_n(s, 10, list(range(measured)))
        qi.measure(s, list(range(measured)))
        s.synchronize()
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] <= 8 << 20
