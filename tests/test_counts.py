"""Tile and share counts at the ends of their ranges (csrc/counts.hpp) on the CPU: arrays of up to 2^31 - 1 elements
and launches of up to 2^32 - 2^16 work units (tests/counts_check.cpp)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT


def test_counts_at_the_ends_of_their_ranges(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "counts_check"
    subprocess.run([cxx, "-std=c++20", "-O1", "-Wall", "-I", os.path.join(PKG_DIR, "csrc"),
                    os.path.join(ROOT, "tests", "counts_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.startswith("ok ")

