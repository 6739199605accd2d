"""A plan whose matrices fit only beside an empty handle cache: the kept handles are given back first."""
import pytest

torch = pytest.importorskip("torch")
from quant_iron_gb300 import workloads  # noqa: E402

pytestmark = pytest.mark.gpu
N = 13


def build(qi, layers):
    plan = qi.Plan(N, qi.F32, workloads.random_circuit(N, layers=layers, seed=2), fusion=qi.FUSION_GREEDY, use_tensor_cores=1)
    k = plan.stats()["n_blocks_by_k"]
    # operand blocks (6 * 4^k floats) and matrices (4^k complex) of the tensor-core blocks, the bulk of a plan
    return plan, sum(32 * 4 ** i * k[i] for i in (5, 6))


def test_cached_handles_are_given_back(qi):
    with qi.DeviceState(N, qi.F32) as s, qi.DeviceState(N, qi.F32) as want:
        s.set_plus()
        small, size = build(qi, 100)
        small.execute(s)
        s.synchronize()
        qi.trim_cache()
        states = [qi.DeviceState(18, qi.F64) for _ in range(15)]   # 4 MiB and a workspace each
        del states
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        room = 256 << 20
        filler = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        free = torch.cuda.mem_get_info()[0]
        slope = (build(qi, 200)[1] - size) / 100.0
        plan, size = build(qi, int(100 + (free + (20 << 20) - size) / slope))
        if not free + (6 << 20) <= size <= free + (40 << 20):
            pytest.skip("the plan's size is not between the memory with and without the cache")
        s.set_plus()
        plan.execute(s)
        got = s.download()
        del filler
        torch.cuda.empty_cache()
        want.set_plus()
        plan.execute(want)
        assert (got == want.download()).all()
