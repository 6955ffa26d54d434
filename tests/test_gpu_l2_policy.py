"""The iteration kernels with and without the evict-first policy (csrc/spmv.cuh, stays_in_l2): 64 iterations
of an LP whose working set lies under the line and of one over it, against the same steps through the
plugin's operations, bit for bit.
"""
import numpy as np
import pytest

import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [290_000, 400_000])
def test_same_steps_as_the_plugin(m):
    lp = g.random_lp(m, seed=m)
    r = ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                         lp.col_upper, algorithm="r2hpdhg", iteration_limit=64, engine={"presolve": False})
    be = ps26119.Backend(lp)
    eta = 0.998 / be.norm2_estimate()
    x, x0, xh, xb = (be.create(False) for _ in range(4))
    y, y0, yh, yb = (be.create(True) for _ in range(4))
    start = np.clip(0.0, be.scaled(3), be.scaled(4))
    be.upload(x, start)
    be.upload(x0, start)
    for k in range(64):
        w = (k + 1.0) / (k + 2.0)
        be.fused_primal(y, x, x0, eta, w, 1.0, xh, xb)
        be.fused_dual(xb, y, y0, eta, w, 1.0, yh, yb)
    s = be.scalars()
    assert r.iterations == 64
    assert np.array_equal(r.x, np.clip(be.scaled(8) * be.download(xh) / s["bound_scale"], lp.col_lower, lp.col_upper))
    assert np.array_equal(r.y, be.scaled(7) * be.download(yh) / s["obj_scale"])
