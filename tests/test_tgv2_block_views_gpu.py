"""The form of TGV2 that runs several iterations per launch, for every count of views that its
kernels are built for (up to 16), against one launch per iteration: u, v, p, q, r, the energy
and the iteration count are equal bit for bit.  test_tgv2_block_rule.py shows without a GPU that
these frames do take that form."""
import numpy as np
import pytest

import mvs_b200 as M

CASES = [
    (57, 41, 2, dict(niters=20, warps=1)),
    (57, 41, 6, dict(niters=20, warps=2)),
    (57, 41, 7, dict(niters=20, warps=1)),
    (160, 120, 8, dict(niters=20, warps=1)),
    (57, 41, 10, dict(niters=20, warps=2)),
    (57, 41, 11, dict(niters=20, warps=1)),
    (160, 120, 12, dict(niters=20, warps=1)),
    (160, 120, 13, dict(niters=20, warps=2)),
    (161, 119, 14, dict(niters=20, warps=1)),
    (200, 150, 15, dict(niters=20, warps=1)),
    (161, 119, 16, dict(niters=50, warps=2, max_iters=71)),
    (160, 120, 16, dict(niters=100, warps=1, tol=4e-3, check_every=20)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,V,kw", CASES)
def test_block_form_for_every_view_count(cuda, w, h, V, kw):
    from test_tgv2_persistent_gpu import _run, _setup
    s = _setup(cuda, w, h, V, seed=w + V)
    a = _run(cuda, s, M.tgv2_params(**kw))
    b = _run(cuda, s, M.tgv2_params(**kw, iteration_kernel=M.TGV2_ITER_LAUNCH))
    assert a[0] == b[0] and a[1] == b[1], (a[:2], b[:2])
    for x, y in zip(a[2:], b[2:]):
        np.testing.assert_array_equal(x, y)
