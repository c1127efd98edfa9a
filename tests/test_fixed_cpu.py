"""The fixed-point group arithmetic of the FP64 form (fixed.cuh) against long
double, compiled for the host with nvcc (no GPU needed): conversions, products,
staple sums, projection, exponentials, and which links it refuses."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_fixed_point_products(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not (os.path.exists(nvcc) or shutil.which("nvcc")):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "fixed_check")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "--expt-relaxed-constexpr", os.path.join(HERE, "fixed_check.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout[-2000:] + out.stderr
