"""The reference-arithmetic sweep divides its projected coordinates by their depth through
one reciprocal and residual corrections.  Its results are bit-exact only if that equals the
IEEE division: compiled from the library's own header, it is compared with a / b over random
operands, over divisors at the ends of a binade, and over quotients next to the middle of two
floats; and a sweep whose homographies are scaled by a power of two (which keeps the IEEE
divisions) gives the same labels and NCC bits."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

import mvs_b200 as M

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent


def test_quotients_equal_ieee_division(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "quot_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false", "-o", str(exe),
                    str(HERE / "cuda" / "quot_check.cu")], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 3, r.stdout + r.stderr
    for line in lines:
        assert ": 0 differences" in line and "no error" in line, line
    assert r.returncode == 0


@pytest.mark.parametrize("win", [3, 7, 11, 15])
def test_scaled_homographies_give_the_same_sweep(cuda, win):
    import torch
    rng = np.random.default_rng(win)
    w, h, V, P = 131, 67, 2, 9
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(cuda)
    ref, srcs = t(rng.uniform(0, 255, (h, w))), t(rng.uniform(0, 255, (V, h, w)))
    H = np.tile(np.eye(3), (V, P, 1, 1))
    H[..., :2, :] += rng.uniform(-0.02, 0.02, (V, P, 2, 3)) * [1, 1, 100]
    H[..., 2, :2] += rng.uniform(-1e-3, 1e-3, (V, P, 2))
    H = H.astype(np.float32)
    d = M.sweep_desc(w, h, V, P, win, M.MOMENTS_REFERENCE, M.SWEEP_PER_VIEW, 1e-4, 0.5, 8.0)
    ws = torch.empty(M.sweep_workspace_bytes(d), dtype=torch.uint8, device=cuda)
    out = []
    for scale in (1.0, 0.25):   # a power of two scales q0, q1, q2 exactly
        depth = torch.empty((h, w), device=cuda)
        labels = torch.empty((V, h, w), dtype=torch.int32, device=cuda)
        best = torch.empty((V, h, w), device=cuda)
        M.sweep(d, ref, srcs, t(H.reshape(V, P, 9) * np.float32(scale)), t(np.linspace(1, 5, P)), depth, labels, best, workspace=ws)
        torch.cuda.synchronize()
        out.append((labels.cpu().numpy(), best.cpu().numpy(), depth.cpu().numpy()))
    assert (out[0][0] >= 0).mean() > 0.5
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
