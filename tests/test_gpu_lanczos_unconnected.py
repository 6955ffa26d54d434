"""The one-launch Lanczos (csrc/lanczos.cuh) on matrices whose columns fall into unconnected parts, near the
most columns that it takes: its blocks are then tied together by nothing but the exchange of their numbers of
runs and the sums, and run far apart from one another. The oracle is the sequential loop; the estimate has
its bits, also when it is repeated and when several of them share the device.
"""
import threading

import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


def parts(shapes, seed):
    """A block-diagonal LP: dense parts of the given rows × columns, in random order along the diagonal."""
    rng = np.random.default_rng(seed)
    rows, cols, m, n = [], [], 0, 0
    for k in rng.permutation(len(shapes)):
        a, b = shapes[k]
        r, c = np.meshgrid(np.arange(a), np.arange(b), indexing="ij")
        rows.append(m + r.ravel()), cols.append(n + c.ravel())
        m, n = m + a, n + b
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    start, index, value = g.csc_from_triplets(m, n, rows, cols, rng.standard_normal(len(rows)))
    full = lambda k, a: np.full(k, float(a))
    return g.Lp(m, n, c=rng.standard_normal(n), col_lower=full(n, 0), col_upper=full(n, 1), row_lower=full(m, -1),
                row_upper=full(m, 1), col_start=start, row_index=index, value=value)


LPS = {
    "diagonal": lambda: parts([(1, 1)] * 40_960, 1),
    "small_parts": lambda: parts([(2, 3)] * 13_000, 2),
    "a_few_long_rows": lambda: parts([(2, 900)] * 8 + [(1, 1)] * 33_000, 3),  # a few blocks are late
    "a_few_columns": lambda: parts([(60, 2)] * 50 + [(1, 1)] * 1_000, 4),
}


@pytest.mark.parametrize("name", list(LPS))
def test_norm_estimate(name):
    lp = LPS[name]()
    want = oracle.Scaled(lp).norm2()
    be = ps26119.Backend(lp)
    assert [be.norm2_estimate() for _ in range(20)] == [want] * 20


@pytest.mark.parametrize("name", list(LPS))
def test_without_cooperative_launches(name, monkeypatch):
    """PS26119_SLAB_VARIANT leaves the kernels' form, for processes in which such a launch would have to wait."""
    monkeypatch.setenv("PS26119_SLAB_VARIANT", "0")
    lp = LPS[name]()
    assert ps26119.Backend(lp).norm2_estimate() == oracle.Scaled(lp).norm2()


def test_estimates_side_by_side():
    lps = [make() for make in LPS.values()]
    want = [oracle.Scaled(lp).norm2() for lp in lps]
    backends = [ps26119.Backend(lp) for lp in lps]
    got = [None] * len(lps)

    def work(k):
        got[k] = [backends[k].norm2_estimate() for _ in range(10)]

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(lps))]
    [t.start() for t in th]
    [t.join() for t in th]
    assert got == [[w] * 10 for w in want]
