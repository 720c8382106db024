"""The contraction walks where their parts meet: the ranks at which the lanes
of a walker, its columns per lane or the walkers per warp change (and ranks
that leave lanes idle), every number of folded levels up to the five that an
8th-order tree allows, chunks of one batch, of less and of more, a last chunk
of one unit, FP32 and BF16 rows. Against the FP64 oracle on the same factor
values; FP32 sums of at most a chunk's products, joined in FP64, stay within
the FP32 bound of the other MTTKRP tests."""
import numpy as np
import pytest

import oracle as O
from _gen import draw_coo

pytestmark = pytest.mark.gpu

TOL_F32 = 2e-5


def rel_err(a, b):
    return float(np.max(np.abs(a - b)) / max(1e-30, np.max(np.abs(b))))


def bf16_values(m):
    b = np.ascontiguousarray(m, dtype=np.float32).view(np.uint32)
    return ((b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32).astype(np.float64)


@pytest.mark.parametrize("R", [1, 4, 5, 8, 9, 16, 17, 31, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("bf16", [False, True])
def test_walks_at_their_edges(gpu, R, bf16):
    A = gpu
    # 8 levels: five hypersparse ones to fold; 3 levels: none or one
    for dims, nnz, seed in (([9, 8, 7, 7, 6, 6, 5, 5], 6001, 3), ([50, 40, 30], 4097, 4)):
        inds, vals, dims = draw_coo(dims, nnz, seed, 0.6)
        ci, cv, cd = O.coo_clean(inds, vals, dims)
        cd = [int(x) for x in cd]
        N = len(cd)
        t = A.Tensor.from_coo(ci, cv, cd)
        _, cands, _ = A.plan_analytic(t, R)
        mats = [np.asarray(m, dtype=np.float32).astype(np.float64) for m in O.init_factors(cd, R, 7)]
        if bf16:
            mats = [bf16_values(m) for m in mats]
        plans = [A.plan_splatt(t, A.CSF_ALLMODE), A.plan_splatt(t, A.CSF_ONEMODE), cands[-1]]
        for plan in plans:
            for chunk in (0, 16, 5, len(cv) - 1):
                e = A.Engine(t, R, plan, bf16=bf16, chunk_leaf=chunk, chunk_rows=chunk)
                e.set_factors(mats)
                for m in range(N):
                    want = O.mttkrp_coo(ci, cv, cd, mats, m, R)
                    assert rel_err(e.mttkrp(m), want) < TOL_F32, (N, m, chunk)
                e.free()
        t.free()


def test_automatic_folds_reach_every_level(gpu):
    """Without a cap, walks over hypersparse trees fold 3, 4 and 5 levels; the
    results repeat bit for bit and stay the oracle's."""
    A = gpu
    for N in (5, 6, 7, 8):
        inds, vals, dims = draw_coo([12, 11, 10, 10, 9, 9, 8, 8][:N], 5000, N, None)
        ci, cv, cd = O.coo_clean(inds, vals, dims)
        cd = [int(x) for x in cd]
        t = A.Tensor.from_coo(ci, cv, cd)
        mats = [np.asarray(m, dtype=np.float32).astype(np.float64) for m in O.init_factors(cd, 32, 1)]
        e = A.Engine(t, 32, A.plan_splatt(t, A.CSF_ALLMODE))
        e.set_factors(mats)
        for m in range(N):
            got = e.mttkrp(m)
            assert rel_err(got, O.mttkrp_coo(ci, cv, cd, mats, m, 32)) < TOL_F32, (N, m)
            assert np.array_equal(got, e.mttkrp(m))
        e.set_deterministic(False)
        for m in range(N):
            assert rel_err(e.mttkrp(m), O.mttkrp_coo(ci, cv, cd, mats, m, 32)) < TOL_F32, (N, m)
        e.free()
        t.free()
