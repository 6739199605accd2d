"""FP32 <psi|H|psi>: sums are folded out of FP32 as often as a sum of one launch per group does it on states of this
size, so terms of one sign do not lose bits to the size of their own sum.

A state of positive amplitudes: every pair of a bond adds with the same sign.  A pair's value c is rounded once, and
once more at the size of its sum: with up to two pairs of FP32 sum the squares of these errors, each a half unit in
the last place at most and 0.58 u c in the mean (u = 2^-24), add up to u^2 sum(c^2) over all pairs.  The root mean
square over the seeds has to be within twice that."""
import numpy as np
import pytest

from quant_iron_gb300 import workloads

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


@pytest.mark.parametrize("kind", ["bonds", "diagonal"])
@pytest.mark.parametrize("n", [10, 13, 16, 20])
def test_terms_of_one_sign(qi, n, kind):
    err, bound = [], []
    for seed in range(6):
        psi = np.random.default_rng(100 * n + seed).uniform(0.5, 1.5, size=1 << n)
        psi = (psi / np.linalg.norm(psi)).astype(np.float32).astype(np.float64)
        i = np.arange(1 << n)
        if kind == "bonds":
            terms = [workloads.term(1.0, [(q, "X"), (q + 1, "X")]) for q in range(n - 1)]
            pairs = [2.0 * psi[i < (i ^ (3 << q))] * psi[(i ^ (3 << q))[i < (i ^ (3 << q))]] for q in range(n - 1)]
        else:
            terms, pairs = [workloads.term(1.0, [])], [psi * psi]
        want = float(np.sum([np.sum(p.astype(np.longdouble)) for p in pairs]))
        with qi.DeviceState(n, qi.F32) as s:
            s.upload(psi)
            err.append(qi.sumop_expectation(s, workloads.terms_array(terms)).real - want)
        bound.append(U * np.sqrt(sum(np.sum(p * p) for p in pairs)))
    assert np.sqrt(np.mean(np.square(err))) <= 2.0 * np.sqrt(np.mean(np.square(bound)))


@pytest.mark.parametrize("n", [5, 9, 10, 12, 16, 19])
def test_diagonal_factors(qi, n):
    """<k|H|k> of fields and ZZ bonds, one amplitude of 1: the factor itself.  The coefficients' larger parts add up
    exactly; the K rests are below 2^-24 S each (S: the coefficients' sum, to a power of two) and their FP32 sums lose
    K 2^-24 of K 2^-24 S at most."""
    rng = np.random.default_rng(n)
    h = rng.uniform(-1.0, 1.0, size=n)
    terms = workloads.terms_array([workloads.term(1.0, [(q, "Z"), (q + 1, "Z")]) for q in range(n - 1)]
                                  + [workloads.term(h[q], [(q, "Z")]) for q in range(n)])
    size = 2.0 ** np.ceil(np.log2(n - 1 + np.sum(np.abs(h))))
    with qi.DeviceState(n, qi.F32) as s:
        for k in rng.integers(0, 1 << n, size=8):
            z = 1.0 - 2.0 * ((int(k) >> np.arange(n)) & 1)
            s.set_basis(int(k))
            e = qi.sumop_expectation(s, terms)
            assert abs(e - (np.sum(z[1:] * z[:-1]) + np.sum(h * z))) <= len(terms) ** 2 * 2.0 ** -48 * size + 1e-14 * size
