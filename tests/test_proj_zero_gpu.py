"""The projections of the iterative solvers keep the sign of a zero component, as the
reference's division does: the library's own header against the IEEE operations, bit for bit."""
import pathlib
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent


def test_projection_keeps_the_sign_of_zero(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "proj_zero_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false", "-o", str(exe),
                    str(HERE / "cuda" / "proj_zero_check.cu")], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 4, r.stdout + r.stderr
    for line in lines:
        assert ": 0 differences" in line and "no error" in line, line
    assert r.returncode == 0
