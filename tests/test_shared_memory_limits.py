"""A kernel's limit on dynamic shared memory is a setting of the process.  Calls on several host
threads each set it before their launches, so it has to be one value for all sizes: a smaller
frame's would have the other threads' launches refused halfway through a run.  The host code runs
here against a recording stand-in for the CUDA runtime."""
import pytest

from fake_cuda import launches, run, shared_memory_limits

FRAMES = "((97, 73), (161, 119), (320, 240), (640, 480))"

SOLVERS = {
    "tvl1_block_kernel": """
for theta in (1.0, 0.5):
    for w, h in %s:
        p = M.tvl1_params(theta=theta)
        M.check(L.mvs_tvl1_denoise(w, h, ptr, ptr, 0.4, 8.0, C.byref(p), ptr, big, None))
""" % FRAMES,
    "sparse_block_kernel": """
for w, h in %s:
    M.check(L.mvs_tgv2_sparse(w, h, ptr, ptr, ptr, 8.0, 100, 2.0, 1.5, 0.02, 1.0, 1.0, 0.0, 1.0, ptr, ptr, big, None))
""" % FRAMES,
    "tgv2_block_kernel": """
f9 = (C.c_float * 144)(*[1, 0, 0, 0, 1, 0, 0, 0, 1] * 16)
for V in (1, 2, 3, 4, 5, 8, 9, 12, 13, 16):
    for w, h in ((97, 73), (160, 120), (320, 240)):
        p = M.tgv2_params(niters=100, warps=1)
        M.check(L.mvs_tgv2_run(w, h, V, ptr, ptr, f9, f9, f9, f9, C.byref(p), 1, 1.0, ptr, None, None, ptr, big, None))
""",
    "tgv2_persistent_kernel": """
f9 = (C.c_float * 144)(*[1, 0, 0, 0, 1, 0, 0, 0, 1] * 16)
for w, h, V in ((640, 480, 8), (600, 420, 3), (320, 240, 4)):
    p = M.tgv2_params(niters=20, warps=1, iteration_kernel=M.TGV2_ITER_PERSISTENT)
    M.check(L.mvs_tgv2_run(w, h, V, ptr, ptr, f9, f9, f9, f9, C.byref(p), 1, 1.0, ptr, None, None, ptr, big, None))
""",
}

NETWORK = {
    "wgrad_tc_kernel": """
for cin in (16, 32, 48, 64, 96, 192):
    for cout in (16, 32, 48, 64, 96, 128, 192):
        for h, w in ((20, 12), (480, 640)):
            M.check(L.mvs_conv3x3_backward(ptr, cin, ptr, ptr, cout, 4, h, w, 0, None, ptr, None, ptr, ptr, 1, None))
""",
}
CALLS = {**SOLVERS, **NETWORK}


@pytest.mark.parametrize("kernel", CALLS)
def test_one_shared_memory_limit_for_all_sizes(kernel):
    log = run(CALLS[kernel])
    limits, seen = shared_memory_limits(log, kernel), launches(log, kernel)
    sizes = {}
    for name, _, _, smem in seen:
        sizes.setdefault(name, set()).add(smem)
    assert max(len(s) for s in sizes.values()) > 1   # the sizes do take different amounts
    for name, s in sizes.items():
        assert len(limits[name]) == 1, (name, limits[name])
        assert max(s) <= max(limits[name])
