"""Builds with another slab size (B200_SLAB_ROWS, csrc/spmv.cuh): the product of Lanczos leaves its tile sums only
where a block is a tile of terms (csrc/reduce.cuh); elsewhere it would write past them. Compiled, not run."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")


@pytest.mark.skipif(not (os.path.exists(NVCC) or shutil.which("nvcc")), reason="no nvcc")
@pytest.mark.parametrize("rows", [128, 256])
def test_tile_sums_only_from_blocks_of_a_tile(rows, tmp_path):
    src = tmp_path / "probe.cu"
    src.write_text('#include "problem.cuh"\nstatic_assert(b200::kLanczosStat == (B200_SLAB_ROWS == 256), "");\n')
    nvcc = NVCC if os.path.exists(NVCC) else "nvcc"
    r = subprocess.run([nvcc, f"-DB200_SLAB_ROWS={rows}", "-std=c++17", "-Xcicc", "-O0", "-Xptxas", "-O0",
                        "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                        os.path.join(ROOT, "ps26119-solver_b200", "csrc"), "-c", str(src), "-o", str(tmp_path / "probe.o")],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
