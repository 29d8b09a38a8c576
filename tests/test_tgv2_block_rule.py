"""Which kernel TGV2 launches for the frames that the GPU tests compare with one launch per
iteration: without this, a change of the rule's constants would leave those tests comparing that
form with itself.  The host code runs against a recording stand-in for the CUDA runtime."""
import pytest

from fake_cuda import launches, run
from test_tgv2_block_views_gpu import CASES

RUN = """
f9 = (C.c_float * 144)(*[1, 0, 0, 0, 1, 0, 0, 0, 1] * 16)
p = M.tgv2_params(**{kw!r})
M.check(L.mvs_tgv2_run({w}, {h}, {V}, ptr, ptr, f9, f9, f9, f9, C.byref(p), 1, 1.0, ptr, None, None, ptr, big, None))
"""


@pytest.mark.parametrize("w,h,V,kw", CASES)
def test_these_frames_take_the_block_form(w, h, V, kw):
    log = run(RUN.format(w=w, h=h, V=V, kw=kw))
    assert not launches(log, "16iteration_kernel")
    names = {name for name, *_ in launches(log, "tgv2_block_kernel")}
    assert len(names) == 1 and f"tgv2_block_kernelILi{(V + 3) // 4 * 4}E" in names.pop()


def test_every_block_kernel_is_covered():
    assert {(V + 3) // 4 * 4 for _, _, V, _ in CASES} == {4, 8, 12, 16}
    assert {13, 14, 15, 16} <= {V for _, _, V, _ in CASES}


@pytest.mark.parametrize("w,h,V,kw", [(640, 480, 8, dict(niters=50, warps=1)),
                                      (320, 240, 4, dict(niters=50, warps=1, iteration_kernel=1))])
def test_large_frames_and_the_launch_form_take_one_launch_per_iteration(w, h, V, kw):
    log = run(RUN.format(w=w, h=h, V=V, kw=kw))
    assert not launches(log, "tgv2_block_kernel")
    assert len(launches(log, "16iteration_kernel")) == 50
