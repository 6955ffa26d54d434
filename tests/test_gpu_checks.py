"""A check's fused kernels (csrc/checks.cuh: k_check_points, k_check_products) through the decisions they
feed, against the oracle, bit for bit in the reference-order mode: iterations, restarts (x, y and the primal
weight follow from them), and the infeasibility verdicts with the ray's objective and violation in their
text. Sizes around the kernels' blocks of 256 columns and rows, and rows of 3, 4, 5 and more entries (four
are gathered together); steps by resident epochs and by the step kernels.
"""
import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu
INF = np.inf


def dense(m, n, per_row, seed):
    rng = np.random.default_rng(seed)
    A = np.zeros((m, n))
    for i in range(m):
        A[i, rng.choice(n, min(n, per_row), replace=False)] = rng.standard_normal(min(n, per_row))
    return A, rng


def feasible(m, n, per_row):
    A, rng = dense(m, n, per_row, m + n)
    x = rng.uniform(0, 1, n)
    lo = np.where(rng.uniform(size=m) < 0.5, A @ x, -INF)
    up = np.where(np.isfinite(lo) & (rng.uniform(size=m) < 0.5), A @ x, A @ x + rng.uniform(0, 1, m))
    return g.from_dense(rng.standard_normal(n), A, lo, up, np.zeros(n), np.where(rng.uniform(size=n) < 0.9, 2.0, 5.0))


def infeasible(m, n, per_row):  # the last two rows contradict each other
    lp = feasible(m - 2, n, per_row)
    A, rng = dense(m, n, per_row, m * n)
    A[m - 1] = A[m - 2]
    b = np.concatenate([lp.row_upper, [1.0, INF]])
    return g.from_dense(rng.standard_normal(n), A, np.concatenate([np.full(m - 1, -INF), [1.5]]), b, np.full(n, -INF),
                        np.full(n, INF))


def unbounded(m, n, per_row):  # one cheap column that no row holds back
    A, rng = dense(m, n, per_row, m * n + 1)
    A[:, n - 1] = np.abs(A[:, n - 1])
    c = rng.uniform(0, 1, n)
    c[n - 1] = -1.0
    return g.from_dense(c, A, A @ np.ones(n) - 1.0, np.full(m, INF), np.zeros(n),
                        np.concatenate([np.full(n - 1, 2.0), [INF]]))


SHAPES = [(3, 4, 2), (255, 257, 3), (256, 256, 4), (257, 255, 5), (300, 513, 9)]


@pytest.mark.parametrize("steps", ["resident", "kernels"])
@pytest.mark.parametrize("kind", [feasible, infeasible, unbounded])
@pytest.mark.parametrize("shape", SHAPES)
def test_decisions_are_the_oracles(shape, kind, steps, monkeypatch):
    if steps == "kernels":
        monkeypatch.setenv("PS26119_SLAB_VARIANT", "0")
    else:
        monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
    lp = kind(*shape)
    r = ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                         lp.col_upper, algorithm="r2hpdhg", iteration_limit=1920,
                         engine={"presolve": False, "exact": True})
    o = oracle.solve(lp, iteration_limit=1920)
    if r.message.startswith("unbounded direction found"):  # the verdict of the solve without an objective
        assert o.message.startswith("unbounded: primal ray")
        o = oracle.solve(lp.with_data(c=np.zeros(lp.num_cols)), iteration_limit=1920)
    if o.status in ("Optimal", "IterationLimit"):
        assert (r.status_name, r.iterations) == (o.status, o.iterations)
        assert np.array_equal(r.x, o.x) and np.array_equal(r.y, o.y) and r.objective == o.objective
    else:
        assert o.message.split(";")[0] in r.message


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", [infeasible, unbounded])
@pytest.mark.parametrize("shape", SHAPES)
def test_pdlp_verdicts_are_certified(shape, kind, precision):
    """PDLP's check: the ray that it reports passes the gate's own certificate check on the host."""
    lp = kind(*shape)
    r = ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                         lp.col_upper, algorithm="pdlp", precision=precision, iteration_limit=64000,
                         engine={"presolve": False})
    assert r.status == (ps26119.INFEASIBLE if kind is infeasible else ps26119.UNBOUNDED), r.message
    assert r.check == "PASS", r.message


@pytest.mark.parametrize("shape", SHAPES)
def test_pdlp_optimum(shape):
    """PDLP's KKT statistics decide when it ends: its optimum is r²HPDHG's, within both tolerances."""
    lp = feasible(*shape)
    args = (lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower, lp.col_upper)
    a, b = (ps26119.solve_lp(*args, algorithm=alg, tolerance=1e-7, engine={"presolve": False}) for alg in ("pdlp", "r2hpdhg"))
    assert a.status == b.status == ps26119.OPTIMAL and a.check == b.check == "PASS"
    assert abs(a.objective - b.objective) <= 1e-6 * (1.0 + abs(b.objective))
