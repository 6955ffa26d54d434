"""The batch's device-side blocks (csrc/batch.cu: k_binterleave, k_isum_seq, k_bfinish_*) at the sizes where
their tiles end: slots around 32 and 64, rows and columns around 32, 64 (a loaded tile) and 192 (three of
them). A scenario's result must not depend on the others in its batch (bit for bit in the reference-order
mode), must be the single-LP engine's up to rounding, and its z must be c − Aᵀy in CSC order.
"""
import numpy as np
import pytest

import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


def model(lp):
    return (lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower, lp.col_upper)


@pytest.mark.parametrize("m,n,K", [(5, 7, 1), (31, 33, 31), (32, 32, 32), (63, 65, 33), (64, 64, 2), (65, 191, 64),
                                   (191, 193, 65), (193, 257, 3)])
def test_scenarios_stand_alone(m, n, K):
    lp = g.random_lp(m, n, nnz_per_row=min(4, n), seed=m + n)
    sc = g.feasible_scenarios(lp, K, seed=K)
    for k in range(0, K, 3):  # some keep the base's vectors, some change the column bounds
        sc[k].pop("obj")
        sc[k]["col_upper"] = np.where(np.arange(n) % 2 == 0, lp.col_upper, lp.col_upper + 1.0)
    opt = {"iteration_limit": 256, "engine": {"exact": True}}
    got = ps26119.solve_batch(*model(lp), scenarios=sc, **opt)
    for k in sorted({0, K // 2, K - 1}):
        one = ps26119.solve_batch(*model(lp), scenarios=[sc[k]], **opt)[0]
        r = got[k]
        assert (r.status, r.iterations, r.objective) == (one.status, one.iterations, one.objective)
        for v in "xyz":
            assert np.array_equal(getattr(r, v), getattr(one, v)), v
        own = lp.with_data(c=sc[k].get("obj", lp.c), row_lower=sc[k]["row_lower"], row_upper=sc[k]["row_upper"],
                           col_upper=sc[k].get("col_upper", lp.col_upper))
        alone = ps26119.solve_lp(*model(own), algorithm="r2hpdhg", iteration_limit=256,
                                 engine={"presolve": False, "exact": True})
        assert alone.iterations == r.iterations
        # 256 iterations of a nonexpansive map: rounding (1e-16 a step and value) stays below 1e-11
        assert np.allclose(r.x, alone.x, rtol=1e-9, atol=1e-10) and np.allclose(r.y, alone.y, rtol=1e-9, atol=1e-10)
        z = own.c.copy()
        for j in range(n):
            for p in range(lp.col_start[j], lp.col_start[j + 1]):
                z[j] -= lp.value[p] * r.y[lp.row_index[p]]
        assert np.array_equal(z, r.z)
