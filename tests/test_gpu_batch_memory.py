"""Device memory of a batch whose slots all end at the same check: the blocks that its iterations need (20 of a
column's and 18 of a row's size) and nothing of that size more for the solutions."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
M, N, W = 20_450, 32_700, 64  # rows and columns whose blocks just fill their size classes of 2 MiB
CODE = f"""
import sys
sys.path.insert(0, {os.path.join(ROOT, "ps26119-solver_b200")!r})
import torch
import ps26119
from ps26119 import generators as g
lp = g.random_lp({M}, {N}, 6, seed=1)
model = (lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower, lp.col_upper)
torch.zeros(1, device="cuda")
ps26119.solve_batch(*model, scenarios=[{{}}], iteration_limit=64)  # the library's code and caches
before = torch.cuda.mem_get_info()[0]
got = ps26119.solve_batch(*model, scenarios=g.feasible_scenarios(lp, {W}, seed=2), iteration_limit=64)
assert all(r.iterations == 64 for r in got)
print(before - torch.cuda.mem_get_info()[0])
"""


def test_solutions_take_no_blocks_of_their_own():
    env = {k: v for k, v in os.environ.items() if k != "PS26119_DEVICE_CACHE_MB"}  # what was allocated stays cached
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr
    taken, block = int(r.stdout), 2 << 20
    column = -(-(8 * N * W + 64) // block) * block
    row = -(-(8 * M * W + 64) // block) * block
    assert taken >= 15 * (column + row)
    # beside them: the scenarios' vectors as they came, sums, tables (less than two column blocks)
    assert taken < 20 * column + 18 * row + 2 * column, (taken, column, row)
