"""Every mode's update and lambda by their definitions, in every form that the
rows after an update take (finished by the update's last block, by one grid, by
two launches), for modes that are not the last as well.

The reference of one update: raw = M V^-1 in FP64 from the factors that the
update read (all are known: the start's, this sweep's and the sweep's before),
lambda = the columns' 2-norms in the first sweep and max(1, column maxima)
after it, the rows raw / lambda.

Bound, row by row in the 2-norm of the raw rows: M is off by at most 2^-20 of
its rows, V by 2^-22 for each of its Grams, the rows by 2^-24, all of which
V^-1 amplifies by at most its condition; lambda is off by as much again. Rows
rounded to BF16: 2^-8 more. Where the condition leaves less than 5% the update is
not looked at."""
import numpy as np
import pytest

import oracle as O
from test_gpu_dense import random_coo

pytestmark = pytest.mark.gpu


def f64(mats):
    return [np.asarray(m, dtype=np.float64) for m in mats]


@pytest.mark.parametrize("R", [1, 5, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("narrow", [False, True])
def test_rows_and_lambda_of_every_mode(gpu, R, narrow):
    A = gpu
    group = 256 // next(lanes for lanes in (4, 8, 16, 32) if R <= 4 * lanes)
    seen = 0
    for rows in (4 * group, 4 * group + 1, 9 * group):
        for place in range(3):
            dims = [90, 80]
            dims.insert(place, rows)
            inds, vals = random_coo(dims, 6000, R + rows + place)
            t = A.Tensor.from_coo(inds, vals, dims)
            plan = A.plan_splatt(t, A.CSF_ALLMODE)
            state, lam = [], []
            for sweeps in range(3):
                e = A.Engine(t, R, plan, bf16=narrow)
                e.init_factors(3)
                if sweeps:
                    e.als(sweeps)
                mats, l = e.get_factors()
                e.free()
                state.append(f64(mats))
                lam.append(l)
            t.free()
            for sweep in (1, 2):
                for m in range(3):
                    read = [state[sweep if k < m else sweep - 1][k] for k in range(3)]
                    M = O.mttkrp_coo(inds, vals, dims, read, m, R)
                    V = np.ones((R, R))
                    for k in range(3):
                        if k != m:
                            V = V * (read[k].T @ read[k])
                    cond = np.linalg.cond(V)
                    bound = 2 * cond * (2.0**-20 + 2 * 2.0**-22 + 2.0**-24)
                    if not bound < 0.05:
                        continue
                    seen += 1
                    raw = np.linalg.solve(V, M.T).T
                    want = np.linalg.norm(raw, axis=0) if sweep == 1 else np.maximum(1.0, raw.max(axis=0))
                    off = np.linalg.norm(state[sweep][m] * want - raw, axis=1)
                    allowed = (bound + (2.0**-8 if narrow else 0.0)) * np.linalg.norm(raw, axis=1)
                    assert np.all(off <= allowed), (dims, sweep, m, cond)
                    if m == 2:
                        assert np.all(np.abs(lam[sweep] - want) <= bound * np.abs(raw).max(axis=0) * np.sqrt(rows)), \
                            (dims, sweep)
    assert seen >= 27, seen
