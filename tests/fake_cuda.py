"""Runs host code of the library against tests/cuda/fake_runtime.c, a stand-in for the
CUDA runtime that only records what it is asked for: no GPU, no torch.

``run(code)`` executes ``code`` in a child process in which ``M`` is the binding, ``L`` its
ctypes library and ``ptr`` a made-up device address, and returns the log's records as lists
of words."""
import pathlib
import subprocess
import sys
import tempfile

HERE = pathlib.Path(__file__).resolve().parent
SMEM_LIMIT = "8"   # cudaFuncAttributeMaxDynamicSharedMemorySize

PRELUDE = """
import ctypes as C, sys
fake = C.CDLL({so!r}, mode=C.RTLD_GLOBAL)
fake.fake_log.restype = C.c_char_p
sys.path.insert(0, {pkg!r})
import numpy as np
import mvs_b200 as M
L = M.lib()
ptr = C.c_void_p(1 << 40)
big = C.c_size_t(1 << 40)
fake.fake_reset()
"""
EPILOGUE = """
sys.stdout.write(fake.fake_log().decode())
"""


def run(code):
    with tempfile.TemporaryDirectory() as tmp:
        so = pathlib.Path(tmp) / "fake_runtime.so"
        subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", "-o", str(so),
                        str(HERE / "cuda" / "fake_runtime.c")], check=True, capture_output=True, text=True)
        pkg = str(HERE.parent / "plane-sweep-cuda_b200")
        r = subprocess.run([sys.executable, "-c", PRELUDE.format(so=str(so), pkg=pkg) + code + EPILOGUE],
                           capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return [line.split() for line in r.stdout.splitlines()]


def launches(log, kernel):
    """(name, grid, threads, dynamic shared memory) of the launches whose kernel's name contains `kernel`."""
    return [(r[1], tuple(map(int, r[2:5])), int(r[5]), int(r[6])) for r in log if r[0] == "launch" and kernel in r[1]]


def shared_memory_limits(log, kernel):
    """{kernel: set of shared-memory limits asked for}"""
    out = {}
    for r in log:
        if r[0] == "attr" and r[2] == SMEM_LIMIT and kernel in r[1]:
            out.setdefault(r[1], set()).add(int(r[3]))
    return out
