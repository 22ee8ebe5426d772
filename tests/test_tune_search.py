"""The autotuner's search (csrc/tune_search.hpp) on made-up probe times: what it applies is never slower than the ordered
kernels' defaults, which are probed first (tests/tune_search_check.cpp)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT


def test_search_on_made_up_times(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "tune_search_check"
    subprocess.run([cxx, "-std=c++20", "-O1", "-Wall", "-I", os.path.join(PKG_DIR, "csrc"),
                    os.path.join(ROOT, "tests", "tune_search_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.startswith("ok ")
