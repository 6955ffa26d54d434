"""The plugin's products launched back to back (csrc/spmv.cuh, k_slab with programmatic dependent launch):
each starts while the one before it ends, and must still see its results. 200 fused steps without a
synchronisation, vectors copied in between, against the oracle's unfused operations, bit for bit. Rows and
columns of less than one slab (256), exactly one, one more, and several; a row of more than a tile (2,048).
"""
import numpy as np
import pytest

import oracle
import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


def long_row(m, n):
    rng = np.random.default_rng(n)
    A = np.where(rng.uniform(size=(m, n)) < 0.01, rng.standard_normal((m, n)), 0.0)
    A[m // 2] = rng.standard_normal(n)
    x = rng.uniform(0, 1, n)
    return g.from_dense(rng.standard_normal(n), A, A @ x, A @ x + 1.0, np.zeros(n), np.full(n, 2.0))


LPS = {"less": lambda: g.random_lp(100, 150, seed=1), "one": lambda: g.random_lp(256, 256, seed=2),
       "one_more": lambda: g.random_lp(257, 513, seed=3), "several": lambda: g.random_lp(3000, seed=4),
       "long_row": lambda: long_row(300, 2500)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(LPS))
def test_chain(name, precision):
    lp = LPS[name]()
    gpu, cpu = ps26119.Backend(lp, exact=True), oracle.Backend(oracle.Scaled(lp))
    got = []
    for b, fused in ((gpu, True), (cpu, False)):
        b.set_precision(precision == "mixed")
        x, x0, xh, xb, gg = (b.create(False) for _ in range(5))
        y, y0, yh, yb, ax = (b.create(True) for _ in range(5))
        b.upload(x, np.sin(1.0 + np.arange(lp.num_cols)))
        b.upload(y, np.cos(2.0 + np.arange(lp.num_rows)))
        for it in range(200):
            w = (it % 40 + 1.0) / (it % 40 + 2.0)
            if it % 40 == 0:
                b.copy(x0, x)
                b.copy(y0, y)
            if fused:
                b.fused_primal(y, x, x0, 0.3, w, 1.0, xh, xb)
                b.fused_dual(xb, y, y0, 0.4, w, 1.0, yh, yb)
            else:
                b.spmv_t(y, gg)
                b.r2h_primal(x, x0, gg, 0.3, w, 1.0, xh, xb)
                b.spmv(xb, ax)
                b.r2h_dual(y, y0, ax, 0.4, w, 1.0, yh, yb)
        got.append([b.download(v) for v in (x, xh, xb, y, yh, yb)] + [b.dot(x, xh), b.norm2(y), b.diff_norm2(xh, x0)])
    for k, (a, b) in enumerate(zip(*got)):
        assert np.array_equal(a, b, equal_nan=True), k
