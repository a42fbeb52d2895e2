"""The loops over a whole row (ks_strided.h) end, and meet every value once, up to rows of 2^32 - 1 values.  On the host: a loop
that wraps is not run on a GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_loops_and_chunks_of_the_longest_rows(tmp_path):
    exe = str(tmp_path / "strided")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "kernel_scheduling_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "strided_main.cpp")], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout
