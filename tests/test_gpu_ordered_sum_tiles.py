"""Reference-order sums around the sizes at which their evaluation changes form: chains added one by
one (up to 1,024 terms), the tile (256), the group of 32 tiles (8,192) and the warp scan over 32
groups (262,144), and inputs whose running sum changes binade in, or at the ends of, a tile. The
oracle is numpy's sequential add.accumulate; equality is bit for bit.
"""
import numpy as np
import pytest

import ps26119

pytestmark = pytest.mark.gpu

SIZES = [1023, 1024, 1025, 1280, 1281, 8191, 8192, 8193, 8448, 262143, 262144, 262145, 270337]


def terms(kind, n):
    rng = np.random.default_rng(n)
    if kind == "positive":
        return rng.uniform(0, 1, n)
    if kind == "drift":  # mixed signs over a slow drift: binades are crossed to and fro
        return rng.standard_normal(n) + 0.05
    if kind == "steps":  # powers of two at the tiles' first and last places, ties elsewhere
        t = rng.choice([0.5, 1.0, 1.5, -0.5], n)
        t[::256] += 2.0 ** rng.integers(0, 40, t[::256].size)
        t[255::256] -= 2.0 ** rng.integers(0, 40, t[255::256].size)
        return t
    t = rng.uniform(0, 1, n)  # returns to zero in the middle of a tile, then goes on
    t[n // 2] = -t[:n // 2].sum()
    return t


@pytest.mark.parametrize("kind", ["positive", "drift", "steps", "return"])
@pytest.mark.parametrize("n", SIZES)
def test_sum_is_sequential(kind, n):
    import torch
    t = terms(kind, n)
    d = torch.as_tensor(t, device="cuda")
    torch.cuda.synchronize()
    seq = lambda a, init: float(np.add.accumulate(np.concatenate([[init], a]))[-1])
    for init in (0.0, 3.0 * 2.0 ** 20):
        assert ps26119.ordered_sum(d.data_ptr(), n, init, "seq").hex() == seq(t, init).hex()
        parts = [seq(t[n * c // 64:n * (c + 1) // 64], 0.0) for c in range(64)]
        assert ps26119.ordered_sum(d.data_ptr(), n, init, "chunk64").hex() == seq(np.array(parts), init).hex()


@pytest.mark.parametrize("kind", ["positive", "drift", "steps", "return"])
@pytest.mark.parametrize("n", [524_288, 524_289, 800_001])
def test_sum_over_rounds_of_groups(kind, n):  # rounds of 32 groups that take turns in two buffers
    import torch
    t = terms(kind, n)
    d = torch.as_tensor(t, device="cuda")
    torch.cuda.synchronize()
    for init in (0.0, 3.0 * 2.0 ** 20):
        want = float(np.add.accumulate(np.concatenate([[init], t]))[-1])
        assert ps26119.ordered_sum(d.data_ptr(), n, init, "seq").hex() == want.hex()
