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
