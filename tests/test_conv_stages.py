"""The convolution's ring takes a third stage only where that costs no wave of resident CTAs: a
deeper ring with fewer CTAs per SM is slower than two stages once the grid is larger than one wave
of them.  The host code runs against a recording stand-in for the CUDA runtime; the launches of a
32-channel input (two slices, so two stages) give the size of two stages."""
import math

import pytest

from fake_cuda import launches, run

SM_BYTES, CTA_BYTES, SMS = 228 * 1024, 1024, 148


def waves(launch):
    _, (gx, gy, gz), _, smem = launch
    return math.ceil(gx * gy * gz / (SMS * min(SM_BYTES // (smem + CTA_BYTES), 6)))


@pytest.mark.parametrize("cout", [16, 32, 48, 64, 96, 128, 192])
def test_no_wave_lost_to_a_deeper_ring(cout):
    shapes = [(b, 480 >> l, 640 >> l) for b in (1, 2, 4) for l in range(4)] + [(1, 20, 12), (1, 375, 1242), (3, 121, 77)]
    log = run(f"""
for B, H, W in {shapes}:
    for cin in (32, 48, 128, 512):
        M.check(L.mvs_conv3x3_forward(ptr, cin, ptr, ptr, {cout}, B, H, W, 1, ptr, ptr, ptr, None))
""")
    conv = launches(log, "conv3x3_tc_kernel")
    assert len(conv) == 4 * len(shapes)
    deeper = 0
    for two, *rest in zip(*[iter(conv)] * 4):
        for one in rest:
            assert one[1] == two[1] and one[3] >= two[3]
            assert waves(one) <= waves(two), (one, two)
            deeper += one[3] > two[3]
    assert deeper   # the third stage is taken where it costs nothing
