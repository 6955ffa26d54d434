"""PS26119_HOST_THREADS=1: solve_batch runs every host pass, the scenarios' fingerprints among them, on the
calling thread, and gives the same fingerprints as with several threads. CPU only: tests/native/batch_threads_check.cpp,
linked with the library's host objects (or compiled from its sources)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_one_host_thread(tmp_path):
    pkg = os.path.join(ROOT, "ps26119-solver_b200")
    csrc = os.path.join(pkg, "csrc")
    units = ("solver.cpp", "certify.cpp", "io.cpp")
    objs = [os.path.join(pkg, "_build", u + ".o") for u in units]
    if not all(os.path.exists(o) for o in objs):
        objs = [os.path.join(csrc, u) for u in units]
    exe = str(tmp_path / "batch_threads_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", csrc, "-I", "/usr/local/cuda/include",
                        os.path.join(ROOT, "tests", "native", "batch_threads_check.cpp"), *objs, "-o", exe, "-lpthread",
                        "-ldl"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr

    def run(threads):
        p = subprocess.run([exe], capture_output=True, text=True, timeout=60,
                           env=dict(os.environ, PS26119_HOST_THREADS=str(threads)))
        assert p.returncode == 0, p.stderr
        lines = p.stdout.split()
        return int(lines[0]), lines[1:]

    started, prints = run(1)
    assert started == 0
    assert len(set(prints)) == 39 and prints[0] == prints[2]  # scenario 2 is the base itself
    if (os.cpu_count() or 1) > 1:
        several, same = run(4)
        assert several > 0 and same == prints
