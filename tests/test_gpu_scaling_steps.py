"""The device's scaling against the oracle's, bit for bit: every sequence of steps (geometric means, Ruiz,
Pock–Chambolle, each with and without the others), over rows and columns of 0 to 7 entries, a full row and
a full column, and entries whose range is wide enough for the geometric means.
"""
import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


def lengths(wide):
    rng = np.random.default_rng(7)
    m, n = 515, 700
    A = np.zeros((m, n))
    for i in range(m):
        A[i, rng.choice(n, i % 8, replace=False)] = 1.0
    A[5], A[:, 11], A[:, 300:340] = 1.0, 1.0, 0.0
    A *= rng.standard_normal((m, n)) * (10.0 ** rng.integers(-6, 6, (m, n)) if wide else 1.0)
    return g.from_dense(rng.standard_normal(n), A, np.full(m, -1.0), np.full(m, 1.0), np.zeros(n), np.ones(n))


@pytest.mark.parametrize("gm", [0, 12])
@pytest.mark.parametrize("ruiz", [0, 1, 2, 10])
@pytest.mark.parametrize("pock", [False, True])
@pytest.mark.parametrize("wide", [False, True])
def test_scaled_problem(gm, ruiz, pock, wide):
    lp = lengths(wide)
    opts = dict(ruiz_iterations=ruiz, pock_chambolle=pock, geometric_mean_iterations=gm,
                geometric_mean_min_log10_range=4.5)
    dev, ref = ps26119.Backend(lp, **opts), oracle.Scaled(lp, **opts)
    for which in range(9):
        assert np.array_equal(dev.scaled(which), ref.get(which)), which
