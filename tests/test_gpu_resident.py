"""Resident epochs (csrc/resident.cuh: one cooperative kernel per epoch, the LP in shared memory) against
the step kernels, which PS26119_SLAB_VARIANT selects: the same bits in every output, for r²HPDHG and PDLP,
fp64 and mixed. The sizes are those at which the kernel's layout changes: fewer columns and rows than
blocks, one element a thread, several, the largest LP that fits and the first that does not; and rows
and columns without entries, a full row, checks every 1 and 7 iterations.
"""
import numpy as np
import pytest

import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


def sparse(m, n, seed, per_row=3, full_row=False):
    """Inequality LP with empty rows and columns (every 7th row, every 5th column)."""
    rng = np.random.default_rng(seed)
    A = np.zeros((m, n))
    for i in range(m):
        if i % 7 != 6:
            A[i, rng.integers(0, n, per_row)] = rng.standard_normal(per_row)
    A[:, 4::5] = 0.0
    if full_row:
        A[0] = rng.standard_normal(n)
    x = rng.uniform(0, 1, n)
    return g.from_dense(rng.standard_normal(n), A, np.full(m, -np.inf), A @ x + rng.uniform(0, 1, m), np.zeros(n),
                        np.full(n, 3.0))


LPS = {
    "1x1": (lambda: g.from_dense([1.0], [[2.0]], [1.0], [4.0], [0.0], [9.0]), 640),
    "3x5": (lambda: sparse(3, 5, 1), 640),
    "70x90": (lambda: sparse(70, 90, 2), 640),
    "full_row": (lambda: sparse(60, 1500, 3, full_row=True), 640),
    "one_each": (lambda: g.random_lp(3001, seed=4), 640),
    "staircase": (lambda: g.staircase_lp(97, seed=5), 640),
    "several_each": (lambda: g.random_lp(61_003, seed=6), 256),
    "largest_fp64": (lambda: g.random_lp(117_000, seed=7), 128),
    "fp32_only": (lambda: g.random_lp(121_000, seed=8), 1280),
    "neither": (lambda: g.random_lp(160_000, seed=8), 128),
}


def solve(lp, K, **kw):
    engine = {"presolve": False, **kw.pop("engine", {})}
    r = ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                         lp.col_upper, sense=lp.sense, iteration_limit=K, engine=engine, **kw)
    return r, ps26119.last_stats()["kernel_launches"]


def same(monkeypatch, lp, K, **kw):
    monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
    a, launches_a = solve(lp, K, **kw)
    monkeypatch.setenv("PS26119_SLAB_VARIANT", "0")
    b, launches_b = solve(lp, K, **kw)
    assert (a.status, a.iterations, a.message) == (b.status, b.iterations, b.message)
    for k in ("objective", "dual_objective", "primal_residual", "dual_residual", "gap"):
        assert np.array_equal(getattr(a, k), getattr(b, k), equal_nan=True), k
    for k in "xyz":
        assert (getattr(a, k) is None) == (getattr(b, k) is None)
        assert getattr(a, k) is None or np.array_equal(getattr(a, k), getattr(b, k)), k
    return launches_a < launches_b


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("algorithm", ["r2hpdhg", "pdlp"])
@pytest.mark.parametrize("name", list(LPS))
def test_same_bits_as_the_step_kernels(name, algorithm, precision, monkeypatch):
    make, K = LPS[name]
    resident = same(monkeypatch, make(), K, algorithm=algorithm, precision=precision)
    assert resident == (name != "neither" and (name != "fp32_only" or precision == "mixed"))


@pytest.mark.parametrize("every", [1, 7])
@pytest.mark.parametrize("algorithm", ["r2hpdhg", "pdlp"])
def test_check_intervals(algorithm, every, monkeypatch):
    lp = g.random_lp(500, seed=9)
    same(monkeypatch, lp, 70, algorithm=algorithm, precision="mixed", engine={"check_every": every})


def test_solves_side_by_side(monkeypatch):
    """Cooperative launches of several threads' solves share the device and do not wait on one another."""
    import threading
    monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
    lps = [g.random_lp(m, seed=m) for m in (700, 9_000, 40_000, 110_000)]
    alone = [solve(lp, 640)[0] for lp in lps]
    got = [None] * len(lps)

    def work(k):
        got[k] = solve(lps[k], 640)[0]

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(lps))]
    [t.start() for t in th]
    [t.join() for t in th]
    for a, b in zip(alone, got):
        assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y) and a.iterations == b.iterations
