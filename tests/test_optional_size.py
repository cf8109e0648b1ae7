"""Device memory that an evaluation can do without (csrc/optional_size.h), by a C++ client with a fake
allocation: what a full GPU would have to show."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_optional_size(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = str(tmp_path / "optional_size")
    src = os.path.join(ROOT, "tests", "cpp", "optional_size.cpp")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-Wextra", "-pthread", src, "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([out], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
