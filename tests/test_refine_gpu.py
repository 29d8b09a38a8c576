"""TGV2, TV-L1 denoise and compute3D on the GPU against the reference and the oracle.

The fused kernels perform the reference's arithmetic statement for statement,
so against the reference's own kernels (golden fixtures, run on the CPU) the
results are bit-identical; against the FP64 oracle the stated bar is 1e-4
relative on the depth.
"""
import numpy as np
import pytest

import pyoracle as po
import mvs_b200 as M
from mvs_b200 import hostmath as hm, scenes

pytestmark = pytest.mark.gpu


def tgv_inputs(g):
    K = g["K"]
    rel = [hm.relative_f32(g["Rref"], g["tref"], g["Rsrc"][i], g["tsrc"][i]) for i in range(len(g["Rsrc"]))]
    invK = hm.inv3_f32(K)
    Rs = np.stack([r[0].reshape(9) for r in rel])
    ts = np.stack([r[1] for r in rel])
    return np.float32(K).reshape(9), invK.reshape(9), Rs, ts


def run_tgv(cuda, ref, srcs, K9, iK9, Rs, ts, params, u0=None):
    import torch
    h, w = ref.shape
    V = len(srcs)
    d_ref = torch.from_numpy(np.ascontiguousarray(ref, np.float32)).to(cuda)
    d_srcs = torch.from_numpy(np.ascontiguousarray(np.stack(srcs), np.float32)).to(cuda)
    u = torch.empty((h, w), dtype=torch.float32, device=cuda)
    if u0 is not None:
        u.copy_(torch.from_numpy(np.ascontiguousarray(u0, np.float32)))
    ws = torch.empty(M.tgv2_workspace_bytes(w, h, V) // 8 + 1, dtype=torch.int64, device=cuda)
    it, e = M.tgv2_run(d_ref, d_srcs, K9, iK9, Rs, ts, params, u, u_from_input=u0 is not None, workspace=ws)
    torch.cuda.synchronize()
    return u.cpu().numpy(), it, e


@pytest.mark.parametrize("name", ["tgv_from_one", "tgv_from_depth"])
def test_tgv2_bit_exact_vs_reference(cuda, golden, name):
    g = golden(name)
    K9, iK9, Rs, ts = tgv_inputs(g)
    p = M.tgv2_params(niters=int(g["niters"]), warps=int(g["warps"]))
    u0 = None if str(g["start"]) == "one" else g["depth_gt"]
    u, it, _ = run_tgv(cuda, g["ref"], list(g["srcs"]), K9, iK9, Rs, ts, p, u0)
    assert it == int(g["niters"]) * int(g["warps"])
    np.testing.assert_array_equal(u, g["u"])


@pytest.mark.parametrize("n_views", [5, 10])
def test_tgv2_view_counts_with_padded_stride_bit_exact(cuda, n_views):
    """The per-view duals and linearisation are stored [pixel][V rounded up to
    4]: 5 views (stride 8, kernel for up to 8 views) and 10 (stride 12, kernel
    for up to 16) equal the oracle's f32 run, which follows the reference's
    arithmetic, bit for bit."""
    fr, planes, win = scenes.config_tiny(seed=9, width=72, height=40, n_src=n_views, n_planes=8, win=5)
    poses = [(c.R, c.t) for c in fr.src_cams]
    K1 = fr.ref_cam.K_1based
    g = dict(K=np.float32(K1), Rref=fr.ref_cam.R, tref=fr.ref_cam.t, Rsrc=np.stack([c.R for c in fr.src_cams]),
             tsrc=np.stack([c.t for c in fr.src_cams]))
    K9, iK9, Rs, ts = tgv_inputs(g)
    u0 = fr.depth_gt.astype(np.float32)
    u, it, _ = run_tgv(cuda, fr.ref, fr.srcs, K9, iK9, Rs, ts, M.tgv2_params(niters=6, warps=2), u0)
    assert it == 12
    uo, _, _ = po.tgv2(fr.ref, fr.srcs, K1, fr.ref_cam.R, fr.ref_cam.t, poses, niters=6, warps=2, u_init=u0,
                       precision="f32")
    np.testing.assert_array_equal(u, uo)


def test_tgv2_anisotropic_tensor_vs_reference(cuda, golden):
    """beta = 1.5, gamma = 0.8: the anisotropic diffusion tensor
    (TGV2_kernels.cu:257-298) weights the P step and the divergence of the U
    step (:300-365).  The tensor is computed with CUDA's expf/powf, the
    reference run on the CPU with the host's: a one-ulp difference of a tensor
    entry moves the depth by far less than 1e-5 relative, so the bar is 1e-5
    (the rest of the arithmetic is the reference's)."""
    g = golden("tgv_aniso")
    K9, iK9, Rs, ts = tgv_inputs(g)
    p = M.tgv2_params(niters=int(g["niters"]), warps=int(g["warps"]), beta=float(g["beta"]), gamma=float(g["gamma"]))
    u, it, _ = run_tgv(cuda, g["ref"], list(g["srcs"]), K9, iK9, Rs, ts, p, g["depth_gt"])
    assert it == int(g["niters"]) * int(g["warps"])
    rel = np.abs(u.astype(np.float64) - g["u"]) / np.abs(g["u"])
    assert rel.max() <= 1e-5, rel.max()
    # the tensor is really on: the isotropic run differs
    u_iso, _, _ = run_tgv(cuda, g["ref"], list(g["srcs"]), K9, iK9, Rs, ts,
                          M.tgv2_params(niters=int(g["niters"]), warps=int(g["warps"])), g["depth_gt"])
    assert np.max(np.abs(u_iso - g["u"]) / np.abs(g["u"])) > 1e-4


def test_tgv2_anisotropic_tensor_through_handle(cuda, golden):
    """The same run through the PlaneSweep handle (PlaneSweep::TGV with beta,
    gamma: planesweep.cpp:381-536), host images in and out."""
    g = golden("tgv_aniso")
    ps = M.PlaneSweep()
    ps.setK(g["K"])
    ps.setNumberofImages(len(g["srcs"]))
    ps.set_reference(g["ref"], g["Rref"], g["tref"])
    ps.set_sources(g["srcs"], g["Rsrc"], g["tsrc"])
    p = M.tgv2_params(niters=int(g["niters"]), warps=int(g["warps"]), beta=float(g["beta"]), gamma=float(g["gamma"]))
    it, _ = ps.TGVext(p, start=2, u_init=g["depth_gt"])
    assert it == int(g["niters"]) * int(g["warps"])
    u = ps.getDepthmapTGV()
    ps.close()
    rel = np.abs(u.astype(np.float64) - g["u"]) / np.abs(g["u"])
    assert rel.max() <= 1e-5, rel.max()


def test_tgv2_tolerance_vs_fp64_oracle(cuda):
    """TGV2 from a noisy start with an energy tolerance: the FP64 oracle stops within one check
    of the GPU, and at the GPU's iteration count the depth and the energy agree within 1e-4
    relative.  (With the reference's step sizes, tau = 0.02 and sigma = 1, the relative
    energy change per 10 iterations stays near 1e-3 for hundreds of iterations, so a 3e-3
    tolerance is used to exercise the stopping rule on a small frame.)"""
    fr, planes, win = scenes.config_tiny(seed=4, width=80, height=60, n_src=3, n_planes=16, win=5)
    rng = np.random.default_rng(4)
    u0 = (fr.depth_gt * (1 + 0.01 * rng.standard_normal(fr.depth_gt.shape))).astype(np.float32)
    poses = [(c.R, c.t) for c in fr.src_cams]
    K1 = fr.ref_cam.K_1based
    g = dict(K=np.float32(K1), Rref=fr.ref_cam.R, tref=fr.ref_cam.t, Rsrc=np.stack([c.R for c in fr.src_cams]),
             tsrc=np.stack([c.t for c in fr.src_cams]))
    K9, iK9, Rs, ts = tgv_inputs(g)
    p = M.tgv2_params(niters=300, warps=1, tol=3e-3, check_every=10)
    u, it, e = run_tgv(cuda, fr.ref, fr.srcs, K9, iK9, Rs, ts, p, u0)
    _, ito, _ = po.tgv2(fr.ref, fr.srcs, K1, fr.ref_cam.R, fr.ref_cam.t, poses, niters=300, warps=1, u_init=u0,
                        precision="f64", tol=3e-3, check_every=10)
    assert 0 < it < 300 and abs(it - ito) <= 10, (it, ito)
    uo, _, eo = po.tgv2(fr.ref, fr.srcs, K1, fr.ref_cam.R, fr.ref_cam.t, poses, niters=it, warps=1, u_init=u0,
                        precision="f64", tol=1e-30, check_every=it)
    assert abs(e - eo[-1]) <= 1e-4 * abs(eo[-1]), (e, eo[-1])
    rel = np.abs(u - uo) / np.abs(uo)
    assert rel.max() <= 1e-4, rel.max()


def test_tvl1_denoise_bit_exact_vs_reference(cuda, golden):
    import torch
    g = golden("tvl1_denoise")
    h, w = g["depth_in"].shape
    d_ref = torch.from_numpy(g["ref"]).to(cuda)
    d = torch.from_numpy(g["depth_in"].copy()).to(cuda)
    ws = torch.empty(M.tvl1_workspace_bytes(w, h) // 8 + 1, dtype=torch.int64, device=cuda)
    M.tvl1_denoise(d_ref, d, float(g["znear"]), float(g["zfar"]), M.tvl1_params(niters=int(g["niters"])), ws)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(d.cpu().numpy(), g["out"])


@pytest.mark.parametrize("w,h,niters,theta", [(2, 2, 1, 1.0), (65, 3, 7, 1.0), (3, 70, 5, 0.5), (56, 24, 4, 1.0),
                                              (57, 41, 13, 1.0), (131, 127, 9, 0.7), (321, 203, 30, 1.0)])
def test_tvl1_denoise_at_region_edges(cuda, w, h, niters, theta):
    """Images around the regions' sizes and iteration counts around the launches' (odd ones
    included), bit for bit against the f32 oracle (beta = 0: no expf / powf in the tensor)."""
    import torch
    rng = np.random.default_rng(w * 1000 + h)
    ref = rng.uniform(0, 255, (h, w)).astype(np.float32)
    depth = rng.uniform(0.5, 5.0, (h, w)).astype(np.float32)
    d = torch.from_numpy(depth.copy()).to(cuda)
    ws = torch.empty(M.tvl1_workspace_bytes(w, h) // 8 + 1, dtype=torch.int64, device=cuda)
    M.tvl1_denoise(torch.from_numpy(ref).to(cuda), d, 0.4, 8.0, M.tvl1_params(niters=niters, theta=theta), ws)
    torch.cuda.synchronize()
    want = po.tvl1_denoise(ref, depth, 0.4, 8.0, niters=niters, theta=theta, precision="f32")
    np.testing.assert_array_equal(d.cpu().numpy(), want)


def test_compute3d_matches_reference(cuda):
    import torch
    fr, _, _ = scenes.config_tiny(seed=6, width=40, height=30, n_src=1)
    L = po.ref_lib()
    K = np.float32(fr.ref_cam.K_1based)
    R = np.float32(fr.ref_cam.R)
    t = np.float32(fr.ref_cam.t)
    depth = fr.depth_gt.copy()
    depth[0, :5] = 7.0                         # beyond the 5.5 cut-off
    # camera -> world as get3Dcoordinates builds it: RelativeMatrices(ref, I)
    Rr, tr = hm.relative_f32(R, t, np.eye(3, dtype=np.float32), np.zeros(3, np.float32))
    d = torch.from_numpy(depth).to(cuda)
    X = torch.zeros_like(d)
    Y = torch.zeros_like(d)
    Z = torch.empty_like(d)
    M.compute3d(d, hm.inv3_f32(K).reshape(9), Rr.reshape(9), tr, X, Y, Z)
    torch.cuda.synchronize()
    o = [np.zeros_like(depth) for _ in range(3)]
    po.oracle_lib().orc_compute3d_f32(40, 30, po._fp(depth), po._fp(hm.inv3_f32(K).reshape(9).copy()),
                                      po._fp(Rr.reshape(9).copy()), po._fp(tr.copy()), *[po._fp(a) for a in o])
    np.testing.assert_array_equal(X.cpu().numpy(), o[0])
    np.testing.assert_array_equal(Y.cpu().numpy(), o[1])
    np.testing.assert_array_equal(Z.cpu().numpy(), o[2])
    if L is not None:   # also the reference's own kernel, when built here
        rx, ry, rz = (np.zeros_like(depth) for _ in range(3))
        L.ref_compute3d(40, 30, po._fp(depth), po._fp(K.reshape(9).copy()), po._fp(R.reshape(9).copy()),
                        po._fp(t.copy()), 0, po._fp(rx), po._fp(ry), po._fp(rz))
        np.testing.assert_array_equal(Z.cpu().numpy(), rz)
