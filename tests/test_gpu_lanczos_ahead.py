"""Lanczos (csrc/problem.cuh) launches no steps past the batch that ends it where a step is expensive: matrices
of nearly rank one, whose estimate ends with the first batch of 21 steps, with long rows or with long columns.
"""
import re

import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(40, 480), (480, 40), (300, 600)])
def test_steps_launched(m, n, capfd):
    rng = np.random.default_rng(m)
    A = np.outer(rng.uniform(0.5, 1.0, m), rng.uniform(0.5, 1.0, n)) + 1e-3 * rng.standard_normal((m, n))
    lp = g.from_dense(rng.uniform(0.0, 1.0, n), A, np.full(m, -1.0), np.full(m, 1.0), np.zeros(n), np.ones(n))
    ps26119.solve_lp(lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower, lp.col_upper,
                     iteration_limit=64, engine={"presolve": False}, verbosity=2)
    out = capfd.readouterr()
    assert [int(k) for k in re.findall(r"Lanczos steps launched: (\d+)", out.out + out.err)] == [21]
    assert ps26119.Backend(lp).norm2_estimate() == oracle.Scaled(lp).norm2()
