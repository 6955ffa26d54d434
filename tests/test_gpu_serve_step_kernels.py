"""Groups of requests that run the grouped step kernels (csrc/spmv.cuh k_group_fed) instead of one resident
launch: because a launch variant is forced, because they do not fit the SMs' shared memory side by side, because
one of them has a row too long for the resident form; and groups that change from one form to the other as
requests leave. Every request's result is that of its own solve, bit for bit.
"""
import numpy as np
import pytest

import ps26119
from ps26119 import generators as g
from test_gpu_resident_long_rows import with_long

pytestmark = pytest.mark.gpu


def served_equals_solo(lps, precisions, limits, slots):
    with ps26119.Server(slots=slots) as srv:
        ids = [srv.submit(lp, precision=p, iteration_limit=k) for lp, p, k in zip(lps, precisions, limits)]
        got = [srv.result(i)[0] for i in ids]
    for lp, p, k, r in zip(lps, precisions, limits, got):
        a = ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower,
                             lp.col_upper, algorithm="r2hpdhg", precision=p, iteration_limit=k)
        assert (r.status, r.iterations, r.message) == (a.status, a.iterations, a.message)
        assert r.objective == a.objective
        for v in "xyz":
            assert np.array_equal(getattr(r, v), getattr(a, v)), v


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_forced_variant(precision, monkeypatch):
    monkeypatch.setenv("PS26119_SLAB_VARIANT", "0")
    lps = [g.random_lp(m, seed=s) for m, s in ((300, 1), (1200, 2), (50, 3), (2500, 4), (800, 5), (150, 6))]
    served_equals_solo(lps, [precision] * len(lps), [20_000] * len(lps), slots=4)


@pytest.mark.parametrize("variant", [None, "0"], ids=["default", "forced"])
def test_both_precisions_in_one_group(variant, monkeypatch):
    if variant is None:
        monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
    else:
        monkeypatch.setenv("PS26119_SLAB_VARIANT", variant)
    lps = [g.random_lp(m, seed=m) for m in (1500, 1600, 1700, 1800, 400, 500)]
    served_equals_solo(lps, ["fp64", "mixed"] * 3, [1920, 2560, 640, 3200, 1280, 2560], slots=6)


def test_form_changes_as_requests_leave(monkeypatch):
    """12 requests of 40,000 rows and columns: six in a group do not fit, the last ones do."""
    monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
    lps = [g.random_lp(16_000, seed=s) for s in range(12)]
    limits = [640 + 320 * k for k in range(12)]
    served_equals_solo(lps, ["fp64", "fp64", "mixed"] * 4, limits, slots=12)


def test_a_long_row_in_the_group(monkeypatch):
    """The requests beside it run step kernels while it is there, and resident epochs before and after."""
    monkeypatch.delenv("PS26119_SLAB_VARIANT", raising=False)
    lps = [g.random_lp(900, seed=1), with_long(g.random_lp(10_000, seed=2), [8_000]), g.random_lp(2_000, seed=3),
           g.random_lp(1_100, seed=4)]
    served_equals_solo(lps, ["fp64"] * 4, [3200, 960, 2560, 640], slots=4)
