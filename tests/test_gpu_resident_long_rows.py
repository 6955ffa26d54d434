"""Resident epochs and the one-launch Lanczos (csrc/resident.cuh, csrc/lanczos.cuh) on LPs with long rows and
columns, which a warp sums together: the bits of the step kernels (PS26119_SLAB_VARIANT selects them) and of
the oracle's norm, at the lengths where the form changes (32 and 64 entries, and the 64 and 128 that a
warp gathers at a time), for one, two and several long rows beside each other and for rows that are all long,
at the sizes of all three block sizes; and the time of an iteration, which one long row must not
make longer than the step kernels' best.
"""
import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g
from test_gpu_resident import same

pytestmark = pytest.mark.gpu


def with_long(lp, lengths, columns=False, seed=1):
    """lp with one more row (or column) of each given number of entries, at random places."""
    rng = np.random.default_rng(seed)
    m, n = lp.num_rows, lp.num_cols
    at = [rng.choice(m if columns else n, k, replace=False) for k in lengths]
    long = np.repeat(np.arange(len(lengths)), lengths)
    rows = np.concatenate([lp.row_index, np.concatenate(at) if columns else m + long])
    cols = np.concatenate([np.repeat(np.arange(n), np.diff(lp.col_start)), n + long if columns else np.concatenate(at)])
    value = np.concatenate([lp.value, rng.uniform(-1.0, 1.0, len(long))])
    more_m, more_n = (0, len(lengths)) if columns else (len(lengths), 0)
    start, index, value = g.csc_from_triplets(m + more_m, n + more_n, rows, cols, value)
    more = lambda a, k, v: np.concatenate([a, np.full(k, v)])
    return g.Lp(m + more_m, n + more_n, c=more(lp.c, more_n, 1.0), col_lower=more(lp.col_lower, more_n, 0.0),
                col_upper=more(lp.col_upper, more_n, 1.0), row_lower=more(lp.row_lower, more_m, -np.inf),
                row_upper=more(lp.row_upper, more_m, 1e4), col_start=start, row_index=index, value=value)


EDGES = [31, 32, 33, 63, 64, 65, 127, 128, 129, 192, 193, 257]
LPS = {
    "edges": lambda: with_long(g.random_lp(700, seed=1), EDGES),  # 256 threads a block
    "edges_columns": lambda: with_long(g.random_lp(700, seed=1), EDGES, columns=True),
    "edges_512": lambda: with_long(g.random_lp(15_000, seed=2), EDGES),
    "edges_1024": lambda: with_long(g.random_lp(40_000, seed=3), EDGES),
    "one": lambda: with_long(g.random_lp(3_000, seed=4), [3_000]),
    "one_column": lambda: with_long(g.random_lp(3_000, seed=4), [2_999], columns=True),
    "two": lambda: with_long(g.random_lp(3_000, seed=5), [2_000, 1_000]),
    "nine": lambda: with_long(g.random_lp(3_000, seed=6), [500] * 9),
    "thirty": lambda: with_long(g.random_lp(3_000, seed=7), [200] * 30),
    "all": lambda: g.random_lp(300, 3_000, 40, seed=8),
    "dense": lambda: g.from_dense(np.ones(90), np.random.default_rng(9).standard_normal((70, 90)), np.full(70, -1.0),
                                  np.full(70, 1.0), np.zeros(90), np.ones(90)),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("algorithm", ["r2hpdhg", "pdlp"])
@pytest.mark.parametrize("name", list(LPS))
def test_same_bits_as_the_step_kernels(name, algorithm, precision, monkeypatch):
    same(monkeypatch, LPS[name](), 320, algorithm=algorithm, precision=precision)


@pytest.mark.parametrize("name", list(LPS))
def test_norm_estimate(name):
    lp = LPS[name]()
    assert ps26119.Backend(lp).norm2_estimate() == oracle.Scaled(lp).norm2()


def test_served_together(monkeypatch):
    """Requests with and without long rows in one launch."""
    monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
    lps = [LPS["edges"](), g.random_lp(900, seed=11), LPS["two"](), LPS["edges_columns"](), g.staircase_lp(10, seed=12)]
    with ps26119.Server(slots=len(lps)) as srv:
        got = [srv.result(i)[0] for i in [srv.submit(lp, iteration_limit=1280) for lp in lps]]
    for lp, r in zip(lps, got):
        a = ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                             lp.col_upper, algorithm="r2hpdhg", iteration_limit=1280)
        assert r.iterations == a.iterations and np.array_equal(r.x, a.x) and np.array_equal(r.y, a.y)


@pytest.mark.parametrize("columns", [False, True], ids=["row", "column"])
@pytest.mark.parametrize("rows,length", [(10_000, 300), (10_000, 3_000), (33_000, 300), (33_000, 3_000)])
def test_time_of_an_iteration(rows, length, columns, monkeypatch):
    """Against the fastest launch variant of the step kernels, with half again as allowance: one thread a long
    row took 1.4 to 12 times that variant's time."""
    lp = with_long(g.random_lp(rows, seed=1), [length], columns)

    def per_iteration(variant):
        if variant is None:
            monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
        else:
            monkeypatch.setenv("PS26119_SLAB_VARIANT", str(variant))
        best = np.inf
        for _ in range(4):
            ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                             lp.col_upper, iteration_limit=256, engine={"presolve": False})
            s = ps26119.last_stats()
            best = min(best, s["spmv_kernel_ms"] / s["spmv_kernel_launches"])
        return best

    assert per_iteration(None) <= 1.5 * min(per_iteration(v) for v in range(7))
