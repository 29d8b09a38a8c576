"""The form of TGV2 that runs several iterations per launch (taken for small frames) against
one launch per iteration: the same operations per pixel, so u, v, p, q, r, the energy and the
iteration count are equal bit for bit, at the edges of its regions, for view counts around
the multiples of four, for counts that are no multiple of a launch's, and where the run stops
at a tolerance or at the cap."""
import numpy as np
import pytest

import mvs_b200 as M
from test_tgv2_persistent_gpu import _run, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,V,kw", [
    (9, 7, 1, dict(niters=5, warps=2)),
    (52, 12, 4, dict(niters=13, warps=1)),
    (61, 33, 5, dict(niters=7, warps=3)),
    (97, 73, 3, dict(niters=30, warps=2, max_iters=41)),
    (161, 119, 9, dict(niters=12, warps=1)),
    (120, 90, 16, dict(niters=9, warps=1)),
    (320, 240, 4, dict(niters=20, warps=2)),
    (160, 120, 5, dict(niters=200, warps=1, tol=3e-3, check_every=10)),
    (128, 96, 4, dict(niters=33, warps=4, tol=4e-3, check_every=7)),
])
def test_block_form_equals_launch_per_iteration(cuda, w, h, V, kw):
    s = _setup(cuda, w, h, V, seed=w)
    a = _run(cuda, s, M.tgv2_params(**kw))
    b = _run(cuda, s, M.tgv2_params(**kw, iteration_kernel=M.TGV2_ITER_LAUNCH))
    assert a[0] == b[0] and a[1] == b[1], (a[:2], b[:2])
    for x, y in zip(a[2:], b[2:]):
        np.testing.assert_array_equal(x, y)
