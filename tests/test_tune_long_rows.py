"""The autotuner's shape classes (csrc/tune.hpp) tell matrices with a long row from those without: a program of
a few lines, compiled here. CPU only."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include <cstdio>
#include "tune.hpp"
using namespace b200;
static bool same(long long a, long long b) {
  const TuneKey x = tune_key(0, 0, 10000, 60000, a), y = tune_key(0, 0, 10000, 60000, b);
  return !(x < y) && !(y < x);
}
int main() {
  const bool ok = same(0, 64) && same(6, 40) && !same(6, 65) && !same(64, 128) && same(65, 127) && !same(127, 128) &&
                  same(2048, 4095) && !same(2048, 4096) && !same(6, 1 << 20);
  std::puts(ok ? "ok" : "failed");
}
"""


def test_a_long_row_is_a_class_of_its_own(tmp_path):
    src, exe = tmp_path / "key.cpp", str(tmp_path / "key")
    src.write_text(SOURCE)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "ps26119-solver_b200", "csrc"), str(src),
                        "-o", exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout.strip() == "ok"
