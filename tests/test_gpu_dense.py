"""The dense half of a sweep where its launches change (few row groups finished
by the update's last block, more by a grid, ranks that take lambda and the Gram
in the rows' launch or in one of their own; the Gram inverse's instances), and
MTTKRP outputs where the sums of cut rows and the zeroing of the output change.

Bounds, for a sweep's last mode, with V the Hadamard of the other modes' Grams
in FP64: the rows satisfy A V = M up to the FP32 MTTKRP's error (2e-5 of its
largest entry, as in the other tests), the Grams' 2^-22 per product and factor
and the rows' own roundings (under 2^-20 per mode of |A| |V| in all), plus
2^-8 of |A| |V| when the rows are rounded to BF16. The fit that the sweep
reports is that of the rows and lambda it leaves, to the 1e-4 of the other
tests."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def random_coo(dims, nnz, seed):
    """Every slice hit, no duplicates."""
    rng = np.random.default_rng(seed)
    inds = np.stack([np.concatenate([np.arange(d), rng.integers(0, d, nnz - d)]) for d in dims]).astype(np.uint64)
    for m in range(1, len(dims)):
        inds[m] = rng.permutation(inds[m])
    inds = np.unique(inds, axis=1)
    return np.ascontiguousarray(inds), rng.random(inds.shape[1]) + 0.1


@pytest.mark.parametrize("R", [1, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("bf16", [False, True])
def test_updates_at_their_edges(gpu, R, bf16):
    A = gpu
    group = 256 // next(lanes for lanes in (4, 8, 16, 32) if R <= 4 * lanes)
    for rows in (1, group, 4 * group, 4 * group + 1, 9 * group):
        for dims in ([60, 50, rows], [rows, 60, 50]):
            inds, vals = random_coo(dims, 4000, R + rows)
            t = A.Tensor.from_coo(inds, vals, dims)
            plan = A.plan_splatt(t, A.CSF_ALLMODE)
            for sweeps in (1, 2):
                e = A.Engine(t, R, plan, bf16=bf16)
                e.init_factors(3)
                res = e.als(sweeps, 0.0)
                mats, lam = e.get_factors()
                e.free()
                mats = [np.asarray(m, dtype=np.float64) for m in mats]
                grams = [m.T @ m for m in mats]
                M = O.mttkrp_coo(inds, vals, dims, mats, 2, R)
                V = grams[0] * grams[1]
                raw = mats[2] * lam
                off = np.abs(raw @ V - M)
                c = 3 * 2.0**-20 + (2.0**-8 if bf16 else 0.0)
                assert np.all(off <= 2e-5 * np.abs(M).max() + c * (np.abs(raw) @ np.abs(V))), (dims, sweeps)
                ttn = float(vals @ vals)
                znorm = float(lam @ (V * grams[2]) @ lam)
                inner = float(np.sum(M * raw))
                fit = 1.0 - np.sqrt(max(0.0, ttn + znorm - 2.0 * inner)) / np.sqrt(ttn)
                # (one row and more columns than it has entries: the residual is
                # lost in ||X||^2 + ||Z||^2 - 2 <X, Z>, a difference of FP32 sums)
                if rows > 1 or R < 50:
                    assert abs(res["fit"] - fit) < 1e-4, (dims, sweeps)
            t.free()


@pytest.mark.parametrize("deterministic", [True, False])
def test_long_chains_of_cut_rows(gpu, deterministic):
    """Two root slices cut into thousands of chunks each, and a leaf row that
    takes a third of the nonzeros: sums over several rounds of 64 groups."""
    A = gpu
    rng = np.random.default_rng(5)
    dims, nnz, R = [2, 700, 900], 300000, 9
    inds = np.unique(np.stack([rng.integers(0, d, nnz) for d in dims]), axis=1)
    inds = np.concatenate([inds, np.stack([inds[0], inds[1], np.zeros_like(inds[2])])], axis=1)
    inds = np.unique(inds, axis=1).astype(np.uint64)
    vals = rng.random(inds.shape[1])
    mats = [np.asarray(m, dtype=np.float32).astype(np.float64) for m in O.init_factors(dims, R, 7)]
    t = A.Tensor.from_coo(inds, vals, dims)
    for flag in (A.CSF_ALLMODE, A.CSF_ONEMODE):
        for chunk in (5, 0):
            e = A.Engine(t, R, A.plan_splatt(t, flag), chunk_leaf=chunk, chunk_rows=chunk)
            e.set_deterministic(deterministic)
            e.set_factors(mats)
            for m in range(3):
                want = O.mttkrp_coo(inds, vals, dims, mats, m, R)
                got = e.mttkrp(m)
                assert np.max(np.abs(got - want)) < 2e-5 * np.max(np.abs(want)), (flag, chunk, m)
                if deterministic:
                    assert np.array_equal(got, e.mttkrp(m))
            e.free()
    t.free()


@pytest.mark.parametrize("deterministic", [True, False])
def test_rows_without_nonzeros_are_zero(gpu, deterministic):
    """Modes with rows that no nonzero has, first, last and between: their
    MTTKRP rows are zero whatever the output buffer held."""
    A = gpu
    rng = np.random.default_rng(6)
    used = [[3, 4, 9], list(range(0, 40, 3)), list(range(5, 30))]
    dims, R = [12, 41, 30], 5
    inds = np.unique(np.stack([rng.choice(u, 500) for u in used]), axis=1).astype(np.uint64)
    vals = rng.random(inds.shape[1])
    mats = [np.asarray(m, dtype=np.float32).astype(np.float64) for m in O.init_factors(dims, R, 7)]
    t = A.Tensor.from_coo(inds, vals, dims)
    for flag in (A.CSF_ALLMODE, A.CSF_ONEMODE):
        e = A.Engine(t, R, A.plan_splatt(t, flag))
        e.set_deterministic(deterministic)
        e.set_factors(mats)
        for m in (0, 1, 2, 1, 0):
            want = O.mttkrp_coo(inds, vals, dims, mats, m, R)
            got = e.mttkrp(m)
            assert np.max(np.abs(got - want)) < 2e-5 * np.max(np.abs(want))
            assert not got[np.setdiff1d(np.arange(dims[m]), used[m])].any()
        e.free()
    t.free()


def test_buffers_kept_for_reuse(gpu):
    """Engines made and freed in turn and on several threads at once compute
    the same sweeps as the first one."""
    import threading

    A = gpu
    inds, vals = random_coo([60, 50, 40], 4000, 1)
    t = A.Tensor.from_coo(inds, vals, [60, 50, 40])
    plan = A.plan_splatt(t, A.CSF_ALLMODE)

    def run(out):
        for R in (8, 24, 8):
            e = A.Engine(t, R, plan)
            e.init_factors(3)
            e.als(3, 0.0)
            out.append(e.get_factors()[0])
            e.free()

    want = []
    run(want)
    got = [[] for _ in range(4)]
    threads = [threading.Thread(target=run, args=(g,)) for g in got]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for g in got:
        assert len(g) == len(want)
        for a, b in zip(g, want):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))
    t.free()
