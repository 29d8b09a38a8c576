"""A reference image of another size set after the sweep: what refines the sweep's depthmap
refuses, before it copies anything (a smaller image would be read past its end, a larger one
would guide the wrong pixels).  The host code runs here against a recording stand-in for the
CUDA runtime."""
import pytest

from fake_cuda import run

SETUP = """
rng = np.random.default_rng(1)

def images(w, h, n=2):
    return rng.uniform(0, 255, (n, h, w)).astype(np.float32)

I, zero = np.eye(3, dtype=np.float32), np.zeros(3, np.float32)

def sources(ps, w, h):
    ps.set_sources(list(images(w, h)), [I, I], [zero, zero])

def swept(w, h):
    ps = M.PlaneSweep()
    ps.set_reference(images(w, h, 1)[0], I, zero)
    sources(ps, w, h)
    ps.setK(I)
    ps.setZ(0.5, 4.0)
    ps.setNumberofImages(2)
    ps.RunAlgorithm()
    return ps

def refused(call):
    fake.fake_reset()
    try:
        call()
    except M.MvsError as e:
        assert e.code == M.MVS_ERR_STATE, e
        assert fake.fake_log() == b"", fake.fake_log()
        return
    raise AssertionError("accepted")
"""


@pytest.mark.parametrize("w,h", [(32, 24), (128, 96), (64, 40), (48, 64)])
def test_denoise_refuses_a_reference_of_another_size(w, h):
    run(SETUP + f"""
ps = swept(64, 48)
ps.CudaDenoise(niters=4)
ps.set_reference(images({w}, {h}, 1)[0], I, zero)
refused(lambda: ps.CudaDenoise(niters=4))
ps.set_reference(images(64, 48, 1)[0], I, zero)   # the sweep's size again
ps.CudaDenoise(niters=4)
""")


@pytest.mark.parametrize("w,h", [(32, 24), (128, 96), (48, 64)])
def test_tgv_refuses_images_of_another_size(w, h):
    run(SETUP + f"""
ps = swept(64, 48)
prm = M.tgv2_params(niters=4, warps=1)
ps.TGVext(prm, start=1)
ps.set_reference(images({w}, {h}, 1)[0], I, zero)
refused(lambda: ps.TGV(niters=4, warps=1))          # the sources are still of the old size
refused(lambda: ps.TGVext(prm, start=0))
sources(ps, {w}, {h})
refused(lambda: ps.TGVext(prm, start=1))            # and the sweep's depthmap is
ps.TGV(niters=4, warps=1)                           # from 1: nothing of the old size
ps.TGVext(prm, start=2, u_init=np.ones(({h}, {w}), np.float32))
ps.RunAlgorithm()
ps.TGVext(prm, start=1)
""")
