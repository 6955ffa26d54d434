"""Solves on several host threads at once and requests on engines of their own: whether an epoch is one resident
launch depends on the solves beside it and changes from epoch to epoch (Engine::epoch_is_resident), the bits
do not; and 16 of them at a time are no slower than by the step kernels (a quarter as allowance), which they
were by 1.9 times when each took its turn on the whole device.
"""
import threading
import time

import numpy as np
import pytest

import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


def solve(lp, **kw):
    return ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                            lp.col_upper, engine={"presolve": False}, **kw)


@pytest.mark.parametrize("algorithm,precision", [("r2hpdhg", "fp64"), ("r2hpdhg", "mixed"), ("pdlp", "fp64")])
def test_same_bits(algorithm, precision):
    lps = [g.random_lp(m, seed=m) for m in (900, 8_000, 10_000, 12_000, 14_000, 16_000)]
    budget = [640 * (k + 1) for k in range(len(lps))]  # they end one after another
    kw = {"algorithm": algorithm, "precision": precision}
    got = [None] * len(lps)

    def one(k):
        got[k] = solve(lps[k], iteration_limit=budget[k], **kw)

    threads = [threading.Thread(target=one, args=(k,)) for k in range(len(lps))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for lp, limit, r in zip(lps, budget, got):
        a = solve(lp, iteration_limit=limit, **kw)
        assert r.iterations == a.iterations and np.array_equal(r.x, a.x) and np.array_equal(r.y, a.y)


def test_time_of_requests_side_by_side(monkeypatch):
    lps = [g.random_lp(m, seed=m) for m in np.geomspace(4_000, 16_000, 16).astype(int)]

    def seconds(variant):
        if variant is None:
            monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
        else:
            monkeypatch.setenv("PS26119_SLAB_VARIANT", variant)
        best = np.inf
        for _ in range(3):
            with ps26119.Server(slots=len(lps), grouped=False) as srv:
                t = time.perf_counter()
                for i in [srv.submit(lp, iteration_limit=12_800) for lp in lps]:
                    srv.result(i)
                best = min(best, time.perf_counter() - t)
        return best

    assert seconds(None) <= 1.25 * seconds("0")
