"""<psi|H|psi> and H|psi> in passes over many X-mask groups: every form a pass takes (and the ones it leaves to
the per-group kernels) against the oracle, at tile edges.

Tolerance, u = 2^-53 or 2^-24, C = sum |c_k|: a term of H|psi> rounds each amplitude by a few u |c_k|, so K terms stay
within 2 (K + 8) u C; an expectation adds up to 200 products in a thread before the FP64 sums, 256 u C."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads
from tests.test_gaterun import random_state

pytestmark = pytest.mark.gpu


def random_terms(n, groups, rng, weight, cplx):
    """Groups of terms sharing X strings of up to `weight` qubits, one to five Z masks each, and diagonal terms."""
    rows = []
    for _ in range(groups):
        x = sum(1 << int(q) for q in rng.permutation(n)[:int(rng.integers(1, min(weight, n) + 1))])
        for _ in range(int(rng.integers(1, 6))):
            z = int(rng.integers(0, 1 << n)) if rng.random() < 0.3 else (x & int(rng.integers(0, 1 << n)))
            rows.append((rng.normal(), rng.normal() if cplx else 0.0, x, z))
    for _ in range(2 * n):
        rows.append((rng.normal(), rng.normal() if cplx else 0.0, 0, int(rng.integers(0, 1 << n))))
    return workloads.terms_array([tuple(r) for r in rows])


def check(qi, orc, n, prec, terms, seed):
    u = 2.0 ** -53 if prec == qi.F64 else 2.0 ** -24
    c = float(np.sum(np.hypot(terms["re"], terms["im"])))
    psi = random_state(n, np.random.default_rng(seed))
    if prec == qi.F32:
        psi = psi.astype(np.complex64).astype(np.complex128)
    with qi.DeviceState(n, prec) as s, qi.DeviceState(n, prec) as out:
        s.upload(psi)
        e = qi.sumop_expectation(s, terms)
        assert abs(e - orc.sumop_expectation(psi, n, terms)) <= 256 * u * c
        qi.sumop_apply(out, s, terms)
        assert np.max(np.abs(out.download() - orc.sumop_apply(psi, n, terms))) <= 2 * (len(terms) + 8) * u * c
        assert np.array_equal(s.download(), psi)


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 9, 10, 11, 12, 13, 15])
def test_random_sums(qi, orc, n, cplx, prec):
    rng = np.random.default_rng(10 * n + cplx)
    check(qi, orc, n, getattr(qi, prec), random_terms(n, 12, rng, 3, cplx), n)
    check(qi, orc, n, getattr(qi, prec), random_terms(n, 6, rng, 6, cplx), n + 50)


@pytest.mark.parametrize("prec", ["F64", "F32"])
@pytest.mark.parametrize("n", [8, 13, 16, 18])
def test_chains_and_lattices(qi, orc, n, prec):
    prec = getattr(qi, prec)
    check(qi, orc, n, prec, workloads.heisenberg_open_chain(n, seed=n), 1)
    check(qi, orc, n, prec, workloads.xxz_periodic(n, seed=n), 2)
    if n % 2 == 0:
        check(qi, orc, n, prec, workloads.lattice_tfim(2, n // 2, seed=n), 3)
