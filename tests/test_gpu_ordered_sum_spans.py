"""Reference-order sums of chains so long that the tiles' approximate sums are added up by spans (csrc/reduce.cuh
k_xspan: more than 12,288 tiles of 256 terms), at the line and around the ends of spans of 1,024 tiles: numpy's
sequential add.accumulate, bit for bit. And their time against that of a chain a quarter as long: without spans the
reads of every block grew with the chain.
"""
import time

import numpy as np
import pytest

import ps26119

pytestmark = pytest.mark.gpu

TILE, SPAN, LINE = 256, 256 * 1024, 256 * 12288


def terms(kind, n):
    rng = np.random.default_rng(n)
    if kind == "positive":
        return rng.uniform(0, 1, n)
    return rng.standard_normal(n) + 0.01  # binades are crossed to and fro


@pytest.mark.parametrize("kind", ["positive", "drift"])
@pytest.mark.parametrize("n", [LINE, LINE + 1, LINE + TILE + 1, 13 * SPAN - 1, 13 * SPAN + 1, 16 * SPAN + 777])
def test_sum_is_sequential(kind, n):
    import torch
    t = terms(kind, n)
    d = torch.as_tensor(t, device="cuda")
    torch.cuda.synchronize()
    want = float(np.add.accumulate(np.concatenate([[3.0], t]))[-1])
    assert ps26119.ordered_sum(d.data_ptr(), n, 3.0, "seq").hex() == want.hex()


def test_chunks_with_spans():
    import torch
    n = 64 * (LINE + 300)  # every one of the 64 chunks has spans
    d = torch.rand(n, dtype=torch.float64, device="cuda")
    t = d.cpu().numpy()
    parts = [float(np.add.accumulate(t[n * c // 64:n * (c + 1) // 64])[-1]) for c in range(64)]
    want = float(np.add.accumulate(np.array(parts))[-1])
    assert ps26119.ordered_sum(d.data_ptr(), n, 0.0, "chunk64").hex() == want.hex()


def test_time_grows_with_the_length():
    import torch
    d = torch.rand(256_000_000, dtype=torch.float64, device="cuda")

    def ms(n):
        best = np.inf
        for _ in range(6):
            torch.cuda.synchronize()
            t = time.perf_counter()
            ps26119.ordered_sum(d.data_ptr(), n)
            best = min(best, time.perf_counter() - t)
        return best

    assert ms(256_000_000) < 7.0 * ms(64_000_000)  # 3.9 with spans, 12 without
