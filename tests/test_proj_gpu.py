"""The iterative solvers form the reference's projections (float)(x / max(1, |x|)) without
the IEEE double square root and divisions.  Their results are bit-exact only if that gives
the same floats: compiled from the library's own header, it is compared with the IEEE
operations over generic and structured values on the GPU."""
import pathlib
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent


def test_projection_equals_ieee_operations(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "proj_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false", "-o", str(exe),
                    str(HERE / "cuda" / "proj_check.cu")], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 7, r.stdout + r.stderr
    for line in lines:
        assert ": 0 differences" in line and "no error" in line, line
    assert r.returncode == 0
