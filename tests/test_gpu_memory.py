"""Device memory of the library: what it keeps for reuse is bounded and goes back
when it is told to."""
import gc

import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def free_bytes():
    import torch
    gc.collect()  # engines of earlier tests that only a cycle holds
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


@pytest.mark.parametrize("deterministic", [True, False])
def test_walks_share_their_scratch(gpu, deterministic):
    """The head and tail rows of a walk's chunks serve all walks of the engine,
    which run one after another, and so do the level sums of the walks below
    the root."""
    A = gpu
    R, chunk = 128, 48  # (one walker per warp: the chunk is a walker's)
    t = A.Tensor.generate([900, 800, 700, 600], 1_500_000, seed=2)
    _, nnz, dims = t.info()
    rows = sum(dims) * R * 4 + max(dims) * R * 8  # factors, MTTKRP rows
    heads_tails = -(-nnz // chunk) * 2 * R * 4
    warm = A.Engine(t, R, A.plan_splatt(t, A.CSF_ALLMODE), chunk_leaf=chunk)
    warm.set_deterministic(deterministic)
    warm.mttkrp(0)
    warm.free()
    for flag in (A.CSF_ALLMODE, A.CSF_ONEMODE):
        A.trim_memory()
        before = free_bytes()
        e = A.Engine(t, R, A.plan_splatt(t, flag), chunk_leaf=chunk)
        e.set_deterministic(deterministic)
        A.trim_memory()
        nfibs = [int(n) for n in e.csf_shape(0)[0]]
        used = before - free_bytes() - sum(e.memory()) - rows
        allowed = 2 * heads_tails + 32 * MIB
        if flag == A.CSF_ONEMODE and deterministic:
            # level sums, and per unit of the levels pulled: order, row, value
            # and its ancestors' rows
            allowed += max(nfibs[1:-1]) * R * 4 + sum(4 * n * (l + 3) for l, n in enumerate(nfibs)) * 2
        elif flag == A.CSF_ONEMODE:
            allowed = sum(nfibs[1:-1]) * R * 4  # less than the two walks' level sums
        e.free()
        assert used <= allowed, (flag, used / MIB, allowed / MIB)
    t.free()


def test_later_walks_leave_captured_sweeps_alone(gpu):
    """A recompute walk made after a sweep was captured needs more scratch than
    the plan's walks; the captured sweep goes on with its own."""
    import numpy as np

    A = gpu
    t = A.Tensor.generate([40, 300, 200, 500], 60000, seed=3)
    plan = [p for p in A.plan_analytic(t, 16)[1] if any(g["n_imten"] for g in p["groups"])][-1]
    want = A.Engine(t, 16, plan)
    want.init_factors(1)
    ref = want.als(3)
    e = A.Engine(t, 16, plan)
    e.init_factors(1)
    e.als_begin(graph=True)
    e.time_sweeps(1)
    for m in range(4):
        a = want.mttkrp_direct(m)
        assert np.array_equal(a, want.mttkrp_direct(m))
        e.mttkrp_direct(m)
    e.time_sweeps(2)
    assert e.fit() == ref["fit"]
    assert all(np.array_equal(x, y) for x, y in zip(e.get_factors()[0], want.get_factors()[0]))
    e.free()
    want.free()
    t.free()
