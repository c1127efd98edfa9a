"""The host loop of the Gauss projection ends on a refused launch, a failed wait and at
its own limit (a fake of the runtime's answers; no GPU needed)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_loop_ends(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "cg_loop_check")
    r = subprocess.run([cxx, "-std=c++17", "-Wall", "-O1", os.path.join(HERE, "cg_loop_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=20)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
