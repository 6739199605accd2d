"""<psi|H|psi> of states whose sums run on less than a warp: every size up to 10 qubits, against numpy in FP64.

Tolerance: up to 2^10 amplitudes and K terms, each product within a few u of |c_k| |psi_i|^2 (u = 2^-53 or 2^-24), and a
sum of 1024 or fewer of them: 256 u sum |c_k|."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from tests.test_gaterun import random_state

pytestmark = pytest.mark.gpu


def expectation(psi, n, terms):
    i, total = np.arange(1 << n), 0.0
    for t in terms:
        x, z = int(t["xmask"]), int(t["zmask"])
        sign = 1.0 - 2.0 * (np.array([bin(int(k) & z).count("1") for k in i]) & 1)
        # P|k> = i^ny (-1)^popc(k & z) |k ^ x>
        total += complex(t["re"], t["im"]) * 1j ** bin(x & z).count("1") * np.vdot(psi[i ^ x], sign * psi)
    return total


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("n", range(1, 11))
def test_against_numpy(qi, n, prec):
    prec = getattr(qi, prec)
    rng = np.random.default_rng(n)
    psi = random_state(n, rng)
    if prec == qi.F32:
        psi = psi.astype(np.complex64).astype(np.complex128)
    rows = [(rng.normal(), 0.0, int(rng.integers(0, 1 << n)) & (3 << k), int(rng.integers(0, 1 << n)))
            for k in range(n) for _ in range(3)]
    terms = workloads.terms_array(rows + [(rng.normal(), 0.0, 0, int(z)) for z in rng.integers(0, 1 << n, size=n)])
    u = 2.0 ** -53 if prec == qi.F64 else 2.0 ** -24
    with qi.DeviceState(n, prec) as s:
        s.upload(psi)
        got = [qi.sumop_expectation(s, t) for t in (terms, terms[:1], terms[-1:])]
    for e, t in zip(got, (terms, terms[:1], terms[-1:])):
        assert abs(e - expectation(psi, n, t)) <= 256 * u * float(np.sum(np.abs(t["re"])))
