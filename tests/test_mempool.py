"""The memory that freed handles leave for the next one (cism_b200/csrc/mempool.h): reuse, bound, return with
the last user and on out-of-memory, and no driver call under its lock.  On a driver of the host's own."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_mempool(tmp_path):
    exe = str(tmp_path / "mempool_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", os.path.join(ROOT, "cism_b200", "csrc"),
                    os.path.join(ROOT, "tests", "mempool_check.cpp"), "-o", exe], check=True, timeout=120)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
