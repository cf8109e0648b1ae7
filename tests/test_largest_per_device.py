"""The per-device shared-memory limit (csrc/largest_per_device.h), by a C++ client with a fake setting:
what a second GPU and threads of different models would have to show."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_largest_per_device(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = str(tmp_path / "largest_per_device")
    src = os.path.join(ROOT, "tests", "cpp", "largest_per_device.cpp")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-Wextra", "-pthread", src, "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([out], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
