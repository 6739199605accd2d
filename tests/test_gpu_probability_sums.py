"""FP32 outcome probabilities: each |a|^2 is rounded to FP32 (twice) and no sum of them is.

A state of positive amplitudes between 0.5 and 1.5: an outcome's sum of M squares, each half a unit in the last place
off at most and 0.58 u of it in the mean (u = 2^-24), is off by 0.58 u / sqrt(M) relative, times 1.2 for the squares'
spread; the total it is normalised by is at least as exact: u / sqrt(M) for the root mean square over outcomes and
seeds.  (FP32 sums of eight squares: 2.4 times the roundings' own error and more.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,measured", [(8, 3), (10, 2), (12, 8), (12, 4), (14, 10), (16, 8), (18, 4)])
def test_outcomes(qi, n, measured):
    err = []
    for seed in range(8):
        rng = np.random.default_rng(10 * n + seed)
        psi = rng.uniform(0.5, 1.5, size=1 << n)
        psi = (psi / np.linalg.norm(psi)).astype(np.float32).astype(np.float64)
        qubits = sorted(int(q) for q in rng.permutation(n)[:measured])
        index = sum(((np.arange(1 << n) >> q) & 1) << k for k, q in enumerate(qubits))
        want = np.bincount(index, weights=psi * psi, minlength=1 << measured)
        with qi.DeviceState(n, qi.F32) as s:
            s.upload(psi)
            _, probs = qi.measure(s, qubits, seed=seed, return_probs=True)
        err.append(probs / (want / want.sum()) - 1.0)
    rest = 2.0 ** (n - measured)
    assert np.sqrt(np.mean(np.square(err))) <= 2.0 ** -24 / np.sqrt(rest) + 1e-15
