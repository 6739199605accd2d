"""set_ghz's second amplitude is in order with what the state's stream does next."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["F64", "F32"])
def test_the_next_call_sees_both_amplitudes(qi, prec):
    n, r = 12, 2.0 ** -0.5
    with qi.DeviceState(n, getattr(qi, prec)) as a, qi.DeviceState(n, getattr(qi, prec)) as b:
        for _ in range(50):
            a.set_ghz()
            b.copy_from(a)
            v = b.download()
            want = np.zeros(1 << n, dtype=complex)
            want[0] = want[-1] = r if prec == "F64" else np.float32(r)
            assert np.array_equal(v, want)
