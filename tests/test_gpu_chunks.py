"""Chunk sizes that a caller names, and the way back to the automatic ones."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walkers", [1, 2])
def test_named_chunks_are_divided_among_the_walkers_set(gpu, walkers):
    """W walkers take a named chunk of W x 64 units in parts of 64, as the W
    walkers that a wider rank has by default do: the FP32 sums of the columns
    that both have are the same ones (another chunk's differ by 1e-8 and more)."""
    A = gpu
    t = A.Tensor.generate([8, 300, 200], 100000, seed=5)
    dims = t.info()[2]
    wide = 128 // walkers  # ranks above 64 and 32: 1 and 2 walkers
    rng = np.random.default_rng(1)
    mats = [rng.random((d, wide), dtype=np.float32).astype(np.float64) for d in dims]
    plan = A.plan_splatt(t, A.CSF_ALLMODE)
    a = A.Engine(t, wide, plan, chunk_leaf=64 * walkers)
    a.set_fold(0)
    a.set_factors(mats)
    b = A.Engine(t, 32, plan, chunk_leaf=64 * walkers)
    b.set_fold(0)
    b.set_walkers(walkers)
    b.set_factors([m[:, :32] for m in mats])
    for m in range(3):
        x, y = a.mttkrp(m)[:, :32], b.mttkrp(m)
        assert np.max(np.abs(x - y)) <= 1e-12 * np.max(np.abs(x)), m
    a.free()
    b.free()
    t.free()


def test_autotuning_can_keep_the_automatic_sizes(gpu):
    """(0, 0) is among the options, and tuning to it alone gives back the engine
    that was there before: every sum, bit for bit."""
    A = gpu
    t = A.Tensor.generate([400, 300, 200, 100], 80000, alpha=1.2, seed=7)
    plan = A.plan_analytic(t, 16)[0]
    mats = O.init_factors(t.info()[2], 16, 3)
    e = A.Engine(t, 16, plan)
    e.set_factors(mats)
    want = [e.mttkrp(m) for m in range(4)]
    e.autotune(((512, 512),), sweeps=1)
    e.set_factors(mats)
    assert not all(np.array_equal(e.mttkrp(m), w) for m, w in enumerate(want))
    assert e.autotune(((0, 0),), sweeps=1) == 0
    e.set_factors(mats)
    assert all(np.array_equal(e.mttkrp(m), w) for m, w in enumerate(want))
    assert e.autotune() in range(5)
    e.free()
    t.free()


def test_default_options_name_the_automatic_sizes():
    import inspect

    import adatm_b200 as A
    assert (0, 0) in inspect.signature(A.Engine.autotune).parameters["options"].default
