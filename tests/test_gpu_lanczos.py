"""The device's Lanczos estimate of the scaled matrix's norm against the oracle's, bit for bit: one
tile of columns, chains added one by one and by tiles, a start vector over many generator jumps, and
a run long enough to reach the host's batches that look ahead.
"""
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu

MODELS = {"one_tile": lambda: g.random_lp(170, seed=2), "one_by_one": lambda: g.random_lp(680, seed=2),
          "tiles": lambda: g.random_lp(700, seed=2), "jumps": lambda: g.random_lp(30_011, seed=2),
          "long": lambda: g.staircase_lp(40, seed=3)}


@pytest.mark.parametrize("name", list(MODELS))
def test_norm_estimate(name):
    lp = MODELS[name]()
    assert ps26119.Backend(lp).norm2_estimate() == oracle.Scaled(lp).norm2()
