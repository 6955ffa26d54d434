"""A check's products on LPs with long rows and columns (csrc/checks.cuh: check_long, from 129 entries on, 64
at a time): the decisions against the oracle, bit for bit in the reference-order mode, for long rows and long
columns, alone in their warp and beside others, for more of them in a warp than it sums together, with the
infeasibility tests' rays; and the time, which one long row must not make longer than by half of what a thread
that walks it alone took (0.17 us an entry).
"""
import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g
from test_gpu_resident_long_rows import with_long

pytestmark = pytest.mark.gpu
INF = np.inf
M, N = 330, 400
EDGES = {3: 129, 5: 257, 40: 128, 70: 192, 71: 193, 100: 320, 328: 320}
MANY = {**{k: 150 for k in range(32, 47)}, **{k: 150 for k in range(64, 80)}}  # 15 in a warp, and 16


def matrix(lengths, columns, seed):
    rng = np.random.default_rng(seed)
    A = np.zeros((N, M) if columns else (M, N))
    for i in range(len(A)):
        at = rng.choice(A.shape[1], lengths.get(i, 3), replace=False)
        A[i, at] = rng.standard_normal(len(at))
    return (A.T.copy() if columns else A), rng


def feasible(A, rng):
    m, n = A.shape
    b = A @ rng.uniform(0, 1, n)
    return g.from_dense(rng.standard_normal(n), A, np.where(rng.uniform(size=m) < 0.5, b, -INF),
                        b + rng.uniform(0, 1, m), np.zeros(n), np.full(n, 2.0))


def infeasible(A, rng):  # the last two rows contradict each other
    m, n = A.shape
    A[m - 1] = A[m - 2]
    lp = feasible(A, rng)
    lower, upper = np.full(m, -INF), lp.row_upper.copy()
    lower[m - 1], upper[m - 2], upper[m - 1] = 1.5, 1.0, INF
    return g.from_dense(lp.c, A, lower, upper, np.full(n, -INF), np.full(n, INF))


def unbounded(A, rng):  # one cheap column that no row holds back
    m, n = A.shape
    A[:, n - 1] = np.abs(A[:, n - 1])
    c = rng.uniform(0, 1, n)
    c[n - 1] = -1.0
    return g.from_dense(c, A, A @ np.ones(n) - 1.0, np.full(m, INF), np.zeros(n), np.concatenate([np.full(n - 1, 2.0), [INF]]))


@pytest.mark.parametrize("kind", [feasible, infeasible, unbounded])
@pytest.mark.parametrize("columns", [False, True], ids=["rows", "columns"])
@pytest.mark.parametrize("lengths", [EDGES, MANY], ids=["edges", "many"])
def test_decisions_are_the_oracles(lengths, columns, kind):
    lp = kind(*matrix(lengths, columns, 7))
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


@pytest.mark.parametrize("columns", [False, True], ids=["row", "column"])
def test_time_of_a_check(columns):
    entries = 60_000
    lp = with_long(g.random_lp(60_000, seed=1), [entries], columns)
    best = INF
    for _ in range(3):
        ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                         lp.col_upper, iteration_limit=640, engine={"presolve": False})
        s = ps26119.last_stats()
        best = min(best, (s["loop_seconds"] * 1e6 - s["spmv_kernel_ms"] * 1e3) / s["checks"])
    assert best <= 0.5 * 0.17 * entries
