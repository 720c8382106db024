"""Device memory of the library: what it keeps for reuse is bounded and goes back
when it is told to."""
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_buffers_go_back(gpu):
    A = gpu
    t = A.Tensor.generate([900, 800, 700, 600], 1_500_000, seed=2)
    plan = A.plan_splatt(t, A.CSF_ALLMODE)
    e = A.Engine(t, 16, plan)  # (kernels loaded, streams made)
    e.init_factors(0)
    first = e.als(1)["fit"]
    e.free()
    A.trim_memory()
    before = free_bytes()
    for _ in range(2):
        e = A.Engine(t, 16, plan)
        e.init_factors(0)
        assert e.als(1)["fit"] == first
        e.free()
        assert before - free_bytes() <= 512 * MIB
    assert before > free_bytes(), "nothing was kept: the test shows nothing"
    A.trim_memory()
    assert free_bytes() == before
    # in use or not, work goes on
    e = A.Engine(t, 16, plan)
    e.init_factors(0)
    A.trim_memory()
    assert e.als(1)["fit"] == first
    e.free()
    t.free()
