"""The device's Lanczos estimate of the scaled matrix's norm against the oracle's, bit for bit: one block
and one run of columns, several, a start vector over many generator jumps, a run long enough to reach the
host's batches that look ahead, the most columns that the resident form takes and one more than that (the
kernels' form), columns and rows without entries, and a full column.
"""
import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu

MODELS = {"one_tile": lambda: g.random_lp(170, seed=2), "one_by_one": lambda: g.random_lp(680, seed=2),
          "tiles": lambda: g.random_lp(700, seed=2), "jumps": lambda: g.random_lp(30_011, seed=2),
          "long": lambda: g.staircase_lp(40, seed=3), "most_columns": lambda: g.random_lp(9_000, 61_440, 6, seed=2),
          "too_many_columns": lambda: g.random_lp(9_000, 61_441, 6, seed=2),
          "most_in_one_launch": lambda: g.random_lp(9_000, 40_960, 6, seed=2),
          "first_past_it": lambda: g.random_lp(9_000, 40_961, 6, seed=2), "holes": lambda: holes(300, 700),
          "one_column": lambda: holes(900, 6)}


def holes(m, n):
    rng = np.random.default_rng(m)
    A = np.where(rng.uniform(size=(m, n)) < 0.02, rng.standard_normal((m, n)), 0.0)
    A[:, n // 2] = rng.standard_normal(m)  # a full column
    A[::5] = 0.0
    A[:, ::3] = 0.0
    return g.from_dense(rng.standard_normal(n), A, np.full(m, -1.0), np.full(m, 1.0), np.zeros(n), np.ones(n))


@pytest.mark.parametrize("name", list(MODELS))
def test_norm_estimate(name):
    lp = MODELS[name]()
    assert ps26119.Backend(lp).norm2_estimate() == oracle.Scaled(lp).norm2()
