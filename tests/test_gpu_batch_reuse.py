"""One BatchSweep used again and again: every round starts from what begin()
computes, and ends bit for bit where a lone engine ends (every sum has an order
of its own, whatever the grids and streams)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows for all three ways to finish an update and to take a Gram: by its last
# block (tens of rows), by a grid (thousands), at ranks below and above 32
SHAPES = [([60, 50, 40], 4000), ([3000, 40, 30, 20], 30000), ([20, 18, 16, 14, 12], 9000), ([2500, 2000, 30], 60000)]


def pairs(A, R):
    out = []
    for k, (dims, nnz) in enumerate(SHAPES):
        t = A.Tensor.generate(dims, nnz, seed=40 + k)
        out.append((t, A.Engine(t, R, A.plan_analytic(t, R)[0])))
    return out


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a[0], b[0])) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("R", [16, 48])
def test_rounds_of_one_batch(gpu, R):
    A = gpu
    rounds = [(0, 1), (1, 2), (2, 1), (0, 1), (3, 3), (4, 1)]  # (seed, sweeps)
    want = []
    for _, e in pairs(A, R):
        got = []
        for seed, sweeps in rounds:
            e.init_factors(seed)
            got.append((e.als(sweeps), e.get_factors()))
        want.append(got)
    batched = pairs(A, R)
    b = A.BatchSweep([e for _, e in batched])
    for k, (seed, sweeps) in enumerate(rounds):
        for _, e in batched:
            e.init_factors(seed)
        b.begin()
        b.time_sweeps(sweeps)
        for (_, e), w in zip(batched, want):
            assert e.fit() == w[k][0]["fit"], k
            assert same(e.get_factors(), w[k][1]), k
    b.free()


def test_engines_changed_between_rounds(gpu):
    """Chunk sizes, walkers, folds and the summation of an engine change after
    its sweep was captured in a batch, which frees what the captured launches
    point to; another batch takes the same engines."""
    A = gpu
    changes = [lambda e: e.autotune(((48, 32),), sweeps=1), lambda e: e.set_walkers(1), lambda e: e.set_fold(0),
               lambda e: (e.set_deterministic(False), e.set_deterministic(True))]
    lone, batched = pairs(A, 16), pairs(A, 16)
    es = [e for _, e in batched]
    b = A.BatchSweep(es)
    for k in range(len(changes) + 1):
        if k:
            changes[k - 1](lone[k - 1][1])
            changes[k - 1](es[k - 1])
        for e in es:
            e.init_factors(k)
        b.begin()
        b.time_sweeps(2)
        for (_, f), e in zip(lone, es):
            f.init_factors(k)
            assert f.als(2)["fit"] == e.fit(), k
            assert same(f.get_factors(), e.get_factors()), k
    # a change between begin and the sweeps, by another batch of the engines
    for e in es:
        e.init_factors(9)
    b.begin()
    other = A.BatchSweep(es[:2])
    b.time_sweeps(2)
    for (_, f), e in zip(lone, es):
        f.init_factors(9)
        assert f.als(2)["fit"] == e.fit()
        assert same(f.get_factors(), e.get_factors())
    other.free()
    b.free()
    with pytest.raises(A.AdatmError):
        A.BatchSweep(es[:1]).time_sweeps(1)
