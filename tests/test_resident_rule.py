"""Which LPs that fit shared memory run resident epochs (csrc/resident_rule.hpp), on the CPU:
tests/native/resident_rule_check.cpp, compiled here. That both forms give the same bits, and that the chosen
one is the faster one, is in tests/test_gpu_resident_long_rows.py."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_resident_rule(tmp_path):
    exe = str(tmp_path / "resident_rule_check")
    src = os.path.join(ROOT, "tests", "native", "resident_rule_check.cpp")
    csrc = os.path.join(ROOT, "ps26119-solver_b200", "csrc")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Wextra", "-I", csrc, src, "-o", exe], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
