"""Rounding of the FP32 walks against FP64, on outputs kept in FP64. The bounds
take every FP32 operation to be off by at most u = 2^-24 of its result and the
errors of different operations to be independent:

* a walker that adds c units in runs of B (16 units, or 32 where two walkers
  share a warp), and the runs' sums to one another, is off by at most
  u sqrt((B^2 + c^2 / B) / 3 / N) of a row of N equal terms (one run of all c
  units: u c / sqrt(3 N));
* the products of a unit are the value's with each row, so units that share
  rows do not share their rounding: u sqrt(k / N) for k products;
* a product of up to three BF16 values is exact, so a value times at most three
  BF16 rows is rounded once."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

U = 2.0**-24


def f32(x):
    return np.asarray(x, dtype=np.float32).astype(np.float64)


def bf16(x):
    b = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32)
    return ((b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32).astype(np.float64)


@pytest.mark.parametrize("R,walkers,run", [(16, 8, 16), (32, 4, 16), (64, 2, 32)])
@pytest.mark.parametrize("narrow", [False, True])
def test_long_runs_of_one_row(gpu, R, walkers, run, narrow):
    A = gpu
    rng = np.random.default_rng(11)
    dims, c = [3, 400, 500], 4096
    inds = np.unique(np.stack([rng.integers(0, d, 360000) for d in dims]), axis=1).astype(np.uint64)
    vals = f32(rng.random(inds.shape[1]) + 0.5)
    mats = [(bf16 if narrow else f32)(rng.random((d, R)) + 0.5) for d in dims]
    t = A.Tensor.from_coo(inds, vals, dims)
    e = A.Engine(t, R, A.plan_splatt(t, A.CSF_ALLMODE), bf16=narrow, chunk_leaf=c * walkers)
    e.set_factors(mats)
    want = O.mttkrp_coo(inds, vals, dims, mats, 0, R)
    off = np.linalg.norm(e.mttkrp(0) - want) / np.linalg.norm(want)
    e.free()
    t.free()
    assert off <= U * np.sqrt((run**2 + c**2 / run) / 3 / (inds.shape[1] / 3))


@pytest.mark.parametrize("R", [16, 32, 64, 128])
def test_units_that_share_rows(gpu, R):
    """All nonzeros of a row have the same leaf and the same parent: a product
    of those two rows alone would be off by the same amount in all of them."""
    A = gpu
    rng = np.random.default_rng(12)
    n = 20000
    dims = [2, n, n + 1, n + 2]
    inds = np.stack([np.arange(n) % 2, np.arange(n), np.full(n, 7), np.full(n, 9)]).astype(np.uint64)
    vals = f32(rng.random(n) + 0.5)
    mats = [f32(rng.random((d, R)) + 0.5) for d in dims]
    t = A.Tensor.from_coo(inds, vals, dims)
    e = A.Engine(t, R, A.plan_splatt(t, A.CSF_ALLMODE))
    e.set_factors(mats)
    want = O.mttkrp_coo(inds, vals, dims, mats, 0, R)
    off = np.linalg.norm(e.mttkrp(0) - want) / np.linalg.norm(want)
    e.free()
    t.free()
    # (20000 units take the smallest chunks: 16 units, one run)
    assert off <= U * (np.sqrt(3 / (n / 2)) + 16 / np.sqrt(3 * n / 2))


@pytest.mark.parametrize("R", [3, 16, 32, 64, 128])
@pytest.mark.parametrize("order", [3, 4])
def test_bf16_rows_round_once(gpu, R, order):
    """One nonzero per output row: from the root of a tree, and from its leaves."""
    A = gpu
    rng = np.random.default_rng(13)
    n = 700
    dims = [n] * order
    inds = np.stack([rng.permutation(n) for _ in dims]).astype(np.uint64)
    vals = f32(rng.random(n) + 0.5)
    mats = [bf16(rng.random((n, R)) + 0.5) for _ in dims]
    t = A.Tensor.from_coo(inds, vals, dims)
    for flag in (A.CSF_ALLMODE, A.CSF_ONEMODE):
        e = A.Engine(t, R, A.plan_splatt(t, flag), bf16=True)
        e.set_factors(mats)
        depth = {int(m): l for l, m in enumerate(e.csf_shape(0)[1])}
        for m in range(order):
            if flag == A.CSF_ONEMODE and 0 < depth[m] < order - 1:
                continue  # summed at its own level first, in FP32
            want = O.mttkrp_coo(inds, vals, dims, mats, m, R)
            got = e.mttkrp(m)
            assert np.max(np.abs(got - want) / want) <= U * (1 + 2.0**-20), (flag, m)
        e.free()
    t.free()
