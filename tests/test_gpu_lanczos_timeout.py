"""A wait that runs out in the one-launch Lanczos (csrc/lanczos.cuh; a limit of no second read makes it run
out) is an error of the call that asked for the estimate, by the plugin, a solve and a batch, and the next
call is as ever: the kernel ends by itself."""
import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


def test_reported_by_every_caller(monkeypatch):
    lp = g.random_lp(3_000, seed=1)
    model = (lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower, lp.col_upper)
    solve = lambda: ps26119.solve_lp(*model, iteration_limit=128, engine={"presolve": False})
    batch = lambda: ps26119.solve_batch(*model, scenarios=[{}, {"obj": 2.0 * lp.c}], iteration_limit=128)
    be = ps26119.Backend(lp)
    want = solve()
    monkeypatch.setenv("PS26119_LANCZOS_POLLS", "0")
    with pytest.raises(RuntimeError, match="timed out"):
        be.norm2_estimate()
    r = solve()
    assert r.status == ps26119.NUMERICAL_ERROR and "timed out" in r.message
    for r in batch():
        assert r.status in (ps26119.NUMERICAL_ERROR, ps26119.NOT_SOLVED) and "timed out" in r.message
    monkeypatch.delenv("PS26119_LANCZOS_POLLS")
    assert be.norm2_estimate() == oracle.Scaled(lp).norm2()
    again = solve()
    assert again.iterations == want.iterations and np.array_equal(again.x, want.x)
    assert all(b.iterations == 128 for b in batch())
