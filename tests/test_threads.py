"""Handles used by several threads at once: the calls of one must not depend on what the
others' lists need (shared memory of the per-subhalo kernel)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_small_and_large_lists_at_the_same_time(tmp_path):
    from hbtplus_gb300 import build
    lib = build.build()
    exe = str(tmp_path / "threads")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "device", "threads.cpp"), lib, "-lpthread",
                    "-Wl,-rpath," + os.path.dirname(lib), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
