"""Workloads of the multiview-stereo engine: what its users have it do, through
its public entry points, over the range of sizes that its configurations,
tests and benchmark use.

    listed()            the standing cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, plans, weights and handles, on the GPU
    run(state)          one pass, and its outputs
    work(case)          the bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64-bit arithmetic, in plain torch

Kinds of case
    sweep    one frame's plane sweep over device tensors, per view or aggregated
    batch    frames of uneven size swept in one graph launch
    handle   a frame from host images to host depthmaps through the PlaneSweep handle
    tgv2     TGV2 multiview refinement of a depthmap
    denoise  TV-L1 depth denoise
    sparse   TGV2 towards a sparse depthmap
    fusion   histogram votes of a depthmap sequence, then TV-L1 fusion
    unet     the warm-start network: prediction, or one training step
"""
import math
import pathlib
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "plane-sweep-cuda_b200"))
import mvs_b200 as M  # noqa: E402
from mvs_b200 import scenes  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # a small frame in the reference's own arithmetic: a robot's or a preview's
        # depthmap, where latency and filling the chip count
        dict(name="sweep small per view", kind="sweep", w=320, h=240, views=4, planes=64, window=7, mode="per_view",
             moments="reference"),
        # the headline frame: precision form, stored BF16 cost volume, winner-take-all over it
        dict(name="sweep frame volume", kind="sweep", w=640, h=480, views=8, planes=256, window=9, mode="aggregated",
             moments="compensated"),
        # a mixed batch: small and full room frames and a street frame of odd width
        dict(name="batch mixed", kind="batch", frames=4, views=6, planes=128, window=0),
        # the drop-in class with its default window and views: host images in, the sweep,
        # the TV-L1 denoise, host depthmaps out
        dict(name="handle frame", kind="handle", w=640, h=480, views=4, planes=128, window=5, iters=100),
        # refinement of a small frame from the reference's constant start, 5 linearisations
        dict(name="tgv2 small", kind="tgv2", w=320, h=240, views=4, iters=20, warps=5, tol=0.0, start="one"),
        # the headline refinement: from the sweep's depth to the energy tolerance
        dict(name="tgv2 frame", kind="tgv2", w=640, h=480, views=8, iters=500, warps=1, tol=1e-4, start="depth"),
        # the denoise between sweep and fusion, its default iteration count
        dict(name="denoise frame", kind="denoise", w=640, h=480, iters=100),
        # densifying a sparse depthmap (5% of the pixels sampled)
        dict(name="sparse frame", kind="sparse", w=640, h=480, iters=200),
        # a small fusion volume of odd sides with the widest histogram: an object scan
        dict(name="fusion small ragged", kind="fusion", vw=100, vh=77, vd=61, bins=10, maps=8, w=320, h=240, iters=50),
        # a room: 256^3 voxels, 40 maps, 200 iterations
        dict(name="fusion room", kind="fusion", vw=256, vh=256, vd=256, bins=7, maps=40, w=640, h=480, iters=200),
        # the warm start of one frame (inference), and its training step
        dict(name="unet predict", kind="unet", w=640, h=480, batch=1, train=False),
        dict(name="unet train", kind="unet", w=640, h=480, batch=4, train=True),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["sweep", "batch", "handle", "tgv2", "denoise", "sparse", "fusion", "unet"])
    w, h = _log(rng, 97, 640), _log(rng, 73, 480)
    if kind == "sweep":
        mode = rng.choice(["per_view", "aggregated"])
        return dict(kind=kind, w=w, h=h, views=rng.randint(2, 8), planes=_log(rng, 16, 256),
                    window=rng.choice([3, 5, 7, 9, 11, 15]), mode=mode,
                    moments=rng.choice(["reference", "compensated"]))
    if kind == "batch":
        return dict(kind=kind, frames=rng.randint(2, 6), views=rng.randint(4, 8), planes=_log(rng, 32, 128),
                    window=rng.choice([0, 5, 9]))
    if kind == "handle":
        return dict(kind=kind, w=w, h=h, views=rng.randint(2, 6), planes=_log(rng, 32, 200),
                    window=rng.choice([3, 5, 7, 9]), iters=rng.randint(20, 100))
    if kind == "tgv2":
        if rng.random() < 0.5:
            return dict(kind=kind, w=w, h=h, views=rng.randint(2, 10), iters=rng.randint(7, 30),
                        warps=rng.randint(2, 8), tol=0.0, start="one")
        return dict(kind=kind, w=w, h=h, views=rng.randint(2, 10), iters=rng.randint(50, 500), warps=1,
                    tol=rng.choice([0.0, 1e-4]), start="depth")
    if kind in ("denoise", "sparse"):
        return dict(kind=kind, w=w, h=h, iters=rng.randint(10, 200))
    if kind == "fusion":
        return dict(kind=kind, vw=_log(rng, 33, 256), vh=_log(rng, 33, 256), vd=_log(rng, 33, 256),
                    bins=rng.randint(2, 10), maps=rng.randint(2, 40), w=320, h=240, iters=rng.randint(10, 200))
    return dict(kind=kind, w=8 * _log(rng, 10, 80), h=8 * _log(rng, 8, 60), batch=rng.randint(1, 4),
                train=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _room(seed, w, h, views):
    """A box room's reference and source views (0..255 grey) and its depth."""
    f = 0.75 * w
    K = scenes.intrinsics(f, f, (w - 1) / 2.0, (h - 1) / 2.0)
    return scenes.GpuRenderer(DEV).frame(seed, w, h, K, views, baseline=(0.02, 0.10))


def _rel(fr):
    return [M.relative_pose(fr.ref_cam.R, fr.ref_cam.t, c.R, c.t) for c in fr.src_cams]


def _gen(seed):
    g = torch.Generator(DEV)
    g.manual_seed(seed)
    return g


def _noisy(depth, seed, lo=0.4, hi=8.0):
    """What a sweep leaves: 1% depth noise and 2% outliers."""
    g = _gen(seed)
    d = depth * (1 + 0.01 * torch.randn(depth.shape, generator=g, device=DEV))
    out = torch.rand(depth.shape, generator=g, device=DEV) < 0.02
    return torch.where(out, lo + (hi - lo) * torch.rand(depth.shape, generator=g, device=DEV), d).clamp(lo, hi).contiguous()


def _planes(n, near=0.4, far=8.0):
    return scenes.inverse_depth_planes(near, far, n)


def _batch_specs(case, seed):
    """Frames in the batch workload's three sizes, in turn."""
    rng = np.random.default_rng(seed)
    kinds = (("room", 640, 480, 481.2, 0.4, 8.0, (0.02, 0.10), 2.0),
             ("street", 1242, 375, 721.5, 2.0, 80.0, (0.05, 0.5), 1.0),
             ("room", 320, 240, 240.0, 0.5, 5.0, (0.05, 0.05), 2.0))
    out = []
    for i in range(case["frames"]):
        scene, w, h, f, near, far, base, rot = kinds[i % 3]
        win = case["window"] or (9, 11, 7, 5)[i % 4]
        out.append(dict(scene=scene, w=w, h=h, K=scenes.intrinsics(f, f, (w - 1) / 2.0, (h - 1) / 2.0), near=near,
                        far=far, base=base, rot=rot, window=win, seed=int(rng.integers(1 << 30)),
                        planes=max(16, case["planes"] >> (i % 2)), views=max(2, case["views"] - i % 3)))
    return out


def _batch_frames(case, seed):
    rnd = scenes.GpuRenderer(DEV)
    frames = []
    for sp in _batch_specs(case, seed):
        fr = rnd.frame(sp["seed"], sp["w"], sp["h"], sp["K"], sp["views"], sp["base"], sp["rot"], sp["scene"])
        frames.append(dict(ref=fr.ref.contiguous(), srcs=fr.srcs, rel=_rel(fr), K1=fr.ref_cam.K_1based,
                           depths=torch.from_numpy(_planes(sp["planes"], sp["near"], sp["far"])).to(DEV),
                           window=sp["window"], zfar=sp["far"],
                           depth=torch.empty((sp["h"], sp["w"]), device=DEV),
                           labels=torch.empty((sp["h"], sp["w"]), dtype=torch.int32, device=DEV),
                           best=torch.empty((sp["h"], sp["w"]), device=DEV)))
    return frames


def _fusion_inputs(case, seed):
    """Noisy depthmaps of the box room along a smooth trajectory (as scenes.fusion_sequence), rendered on the GPU."""
    rng = np.random.default_rng(seed)
    sc = scenes.box_room(seed)
    w, h = case["w"], case["h"]
    f = 0.75 * w
    K = scenes.intrinsics(f, f, (w - 1) / 2.0, (h - 1) / 2.0)
    phase = rng.uniform(0, 2 * math.pi)
    cams = []
    for i in range(case["maps"]):
        a = phase + 0.9 * i / max(case["maps"] - 1, 1)
        c = np.array([0.8 * math.sin(a), -0.3 + 0.1 * math.sin(2 * a), -1.6 + 0.4 * math.cos(a)])
        R, t = scenes.look_at(c, np.array([0.3 * math.sin(a + 1.0), 0.3, 2.0]))
        cams.append(scenes.Camera(K, R, t, w, h))
    _, depth = scenes.GpuRenderer(DEV).render(sc, cams, with_image=False)
    Ks = np.stack([c.K for c in cams]).astype(np.float32)
    Rs = np.stack([c.R for c in cams]).astype(np.float32)
    ts = np.stack([c.t for c in cams]).astype(np.float32)
    a, b = np.array([-2.5, -1.5, -2.5], np.float32), np.array([2.5, 3.5, 2.5], np.float32)
    return _noisy(depth, seed, 0.3, 6.0), Ks, Rs, ts, a, b


def _unet_params(seed):
    """He-normal weights as Unet.init_params makes them, with small biases and a head
    that moves the depth: layers' W[cout][cin][3][3] and b[cout], then the head's."""
    rng = np.random.default_rng(seed)
    parts = []
    for l, (ci, co) in enumerate(M.UNET_LAYERS):
        wt = rng.standard_normal((co, ci, 9)) * math.sqrt(2.0 / (9 * (3 if l == 0 else ci)))
        if l == 0:
            wt[:, 3:, :] = 0.0
        parts += [wt.reshape(-1), rng.standard_normal(co) * 0.01]
    parts += [rng.standard_normal(48) * 0.01, np.zeros(3)]
    return np.concatenate(parts).astype(np.float32)


def _unet_inputs(case, seed):
    w, h, B = case["w"], case["h"], case["batch"]
    fr = [_room(seed * 16 + k, w, h, 1) for k in range(B)]
    gt = torch.stack([f.depth_gt for f in fr])
    g = _gen(seed + 1)
    return dict(ref=torch.stack([f.ref for f in fr]).contiguous(), wta=_noisy(gt, seed),
                cost=torch.rand(gt.shape, generator=g, device=DEV), ut=gt.contiguous(),
                vt=(0.01 * torch.randn((B, 2, h, w), generator=g, device=DEV)).contiguous())


def _sparse_samples(depth, seed):
    g = _gen(seed + 2)
    return torch.where(torch.rand(depth.shape, generator=g, device=DEV) < 0.05, depth, torch.zeros_like(depth)).contiguous()


def _workspace(nbytes):
    return torch.empty(max(int(nbytes), 256), dtype=torch.uint8, device=DEV)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    k = case["kind"]
    s = dict(case=case)
    if k == "sweep":
        fr = _room(seed, case["w"], case["h"], case["views"])
        per_view = case["mode"] == "per_view"
        n = (case["h"], case["w"])
        d = M.sweep_desc(case["w"], case["h"], case["views"], case["planes"], case["window"],
                         M.MOMENTS_REFERENCE if case["moments"] == "reference" else M.MOMENTS_COMPENSATED,
                         M.SWEEP_PER_VIEW if per_view else M.SWEEP_AGGREGATED, 1e-4, 0.5, 8.0)
        volume = not per_view and case["w"] * case["h"] % 8 == 0   # winner-take-all over a stored volume
        out = (case["views"],) + n if per_view else n
        s.update(desc=d, ref=fr.ref.contiguous(), srcs=fr.srcs, K=fr.ref_cam.K_1based, rel=_rel(fr),
                 depths=torch.from_numpy(_planes(case["planes"])).to(DEV),
                 H=torch.empty((case["views"], case["planes"], 9), device=DEV), depth=torch.empty(n, device=DEV),
                 labels=torch.empty(out, dtype=torch.int32, device=DEV), best=torch.empty(out, device=DEV),
                 cost=torch.empty((case["planes"],) + n, dtype=torch.bfloat16, device=DEV) if volume else None,
                 ws=_workspace(M.sweep_workspace_bytes(d)))
    elif k == "batch":
        s["frames"] = _batch_frames(case, seed)
        s["batch"] = M.Batch(s["frames"], M.MOMENTS_COMPENSATED, (64, 3, M.BATCH_ORDER_FRAME, 0))
    elif k == "handle":
        fr = _room(seed, case["w"], case["h"], case["views"])
        ps = M.PlaneSweep()
        ps.setK(fr.ref_cam.K_1based.astype(np.float32))
        ps.setZ(0.4, 8.0)
        ps.setPlaneDepths(_planes(case["planes"]))
        ps.setWindowSize(case["window"])
        ps.setNumberofImages(case["views"])
        n = (case["h"], case["w"])
        s.update(ps=ps, ref=fr.ref.cpu().numpy(), srcs=fr.srcs.cpu().numpy(),
                 R0=fr.ref_cam.R.astype(np.float32), t0=fr.ref_cam.t.astype(np.float32),
                 R=np.stack([c.R for c in fr.src_cams]).astype(np.float32),
                 t=np.stack([c.t for c in fr.src_cams]).astype(np.float32),
                 depth=np.empty(n, np.float32), denoised=np.empty(n, np.float32), gray=np.empty(n, np.uint8))
    elif k == "tgv2":
        fr = _room(seed, case["w"], case["h"], case["views"])
        K, invK, R, t = M.float_cams(fr.ref_cam.K_1based, _rel(fr))
        s.update(ref=fr.ref.contiguous(), srcs=fr.srcs, K=K, invK=invK, R=R, t=t, start=_noisy(fr.depth_gt, seed),
                 u=torch.empty_like(fr.depth_gt).contiguous(),
                 prm=M.tgv2_params(niters=case["iters"], warps=case["warps"], tol=case["tol"]),
                 ws=_workspace(M.tgv2_workspace_bytes(case["w"], case["h"], case["views"])))
    elif k == "denoise":
        fr = _room(seed, case["w"], case["h"], 1)
        s.update(ref=fr.ref.contiguous(), start=_noisy(fr.depth_gt, seed), depth=torch.empty_like(fr.depth_gt),
                 prm=M.tvl1_params(niters=case["iters"]), ws=_workspace(M.tvl1_workspace_bytes(case["w"], case["h"])))
    elif k == "sparse":
        fr = _room(seed, case["w"], case["h"], 1)
        s.update(ref=fr.ref.contiguous(), depth=_noisy(fr.depth_gt, seed), sparse=_sparse_samples(fr.depth_gt, seed),
                 out=torch.empty_like(fr.depth_gt), ws=_workspace(M.tgv2_sparse_workspace_bytes(case["w"], case["h"])))
    elif k == "fusion":
        depth, K, R, t, a, b = _fusion_inputs(case, seed)
        s.update(maps=depth, K=K, R=R, t=t, vol=M.FusionVolume((case["vw"], case["vh"], case["vd"]), case["bins"], a, b))
    else:
        s.update(_unet_inputs(case, seed))
        net = M.Unet(case["batch"], case["h"], case["w"])
        net.set_params(_unet_params(seed))
        s.update(net=net, u=torch.empty_like(s["wta"]), v=torch.empty_like(s["vt"]))
    return s


class _DeviceArray:
    """A device pointer of the engine's, for torch to look at in place.  The
    tensor keeps this object, and this object its owner, so the memory outlives
    the tensor."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3)


def _view(owner, ptr, shape, typestr):
    return torch.as_tensor(_DeviceArray(ptr, shape, typestr, owner), device=DEV)


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "sweep":
        M.sweep_homographies(s["desc"], s["K"], s["rel"], s["depths"], s["H"])
        if s["cost"] is None:
            M.sweep(s["desc"], s["ref"], s["srcs"], s["H"], s["depths"], s["depth"], s["labels"], s["best"],
                    workspace=s["ws"])
            return dict(depth=s["depth"], labels=s["labels"], best=s["best"])
        M.sweep(s["desc"], s["ref"], s["srcs"], s["H"], s["depths"], s["depth"], cost=s["cost"], workspace=s["ws"])
        M.sweep_wta_volume(s["cost"], s["depths"], case["w"] * case["h"], case["planes"], 8.0, s["depth"], s["labels"],
                           s["best"])
        return dict(depth=s["depth"], labels=s["labels"], best=s["best"], cost=s["cost"])
    if k == "batch":
        s["batch"].run()
        return [dict(depth=f["depth"], labels=f["labels"], best=f["best"]) for f in s["frames"]]
    if k == "handle":
        ps = s["ps"]
        ps.set_reference(s["ref"], s["R0"], s["t0"])
        ps.set_sources(s["srcs"], s["R"], s["t"])
        ps.RunAlgorithm()
        ps.CudaDenoise(niters=case["iters"])
        return dict(depth=ps.getDepthmap(out=s["depth"]), denoised=ps.getDepthmapDenoised(out=s["denoised"]),
                    gray=ps.getDepthmap8uDenoised(out=s["gray"]))
    if k == "tgv2":
        if case["start"] == "depth":
            s["u"].copy_(s["start"])
        iters, _ = M.tgv2_run(s["ref"], s["srcs"], s["K"], s["invK"], s["R"], s["t"], s["prm"], s["u"],
                              u_from_input=case["start"] == "depth", workspace=s["ws"])
        return dict(u=s["u"], iters=iters)
    if k == "denoise":
        s["depth"].copy_(s["start"])
        M.tvl1_denoise(s["ref"], s["depth"], 0.4, 8.0, s["prm"], s["ws"])
        return dict(depth=s["depth"])
    if k == "sparse":
        M.tgv2_sparse(s["ref"], s["depth"], s["sparse"], 8.0, s["out"], s["ws"], case["iters"])
        return dict(depth=s["out"])
    if k == "fusion":
        vol = s["vol"]
        vol.reset()
        vol.histogram(s["maps"], s["K"], s["R"], s["t"], 0.05)
        vol.tvl1(case["iters"], 0.1, 0.5, 1.0)
        d, n = vol.device_state(), vol.n
        return dict(u=_view(vol, d["u"], (n,), "<f4"), v=_view(vol, d["v"], (n,), "<f4"), p=_view(vol, d["p"], (3, n), "<f4"),
                    hist=_view(vol, d["hist"], (n, d["hist_stride"]), "<i2"))
    if not case["train"]:
        s["net"].forward(s["wta"], s["cost"], s["ref"], s["u"], s["v"])
        return dict(u=s["u"], v=s["v"])
    loss = s["net"].train_step(s["wta"], s["cost"], s["ref"], s["ut"], s["vt"], 1e-4)
    _, grads = s["net"].get_params(grads=True)
    return dict(loss=np.float32(loss), grads=grads)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

_UNET_LEVEL = (0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0)


def work(case):
    """Each input read once and each output written once; operations of the
    algorithm: 50 per NCC evaluation, and per pixel or voxel and iteration the
    additions, products and comparisons of the update."""
    k = case["kind"]
    if k in ("sweep", "handle"):
        n = case["w"] * case["h"]
        V, P = case["views"], case["planes"]
        by, fl = 4 * n * (1 + V) + 4 * P, 50 * n * V * P
        if k == "handle":
            return dict(bytes=by + 9 * n, flops=fl + 45 * n * case["iters"])
        if case["mode"] == "per_view":
            return dict(bytes=by + 4 * n * (1 + 2 * V), flops=fl)
        volume = 2 * n * P if n % 8 == 0 else 0
        return dict(bytes=by + 12 * n + volume, flops=fl)
    if k == "batch":
        by = fl = 0
        for sp in _batch_specs(case, 0):
            n = sp["w"] * sp["h"]
            by += 4 * n * (1 + sp["views"]) + 12 * n
            fl += 50 * n * sp["views"] * sp["planes"]
        return dict(bytes=by, flops=fl)
    if k == "tgv2":
        n, V = case["w"] * case["h"], case["views"]
        return dict(bytes=4 * n * (1 + V) + 8 * n, flops=n * case["warps"] * (case["iters"] * (100 + 9 * V) + 150 * V))
    if k == "denoise":
        n = case["w"] * case["h"]
        return dict(bytes=12 * n, flops=45 * n * case["iters"])
    if k == "sparse":
        n = case["w"] * case["h"]
        return dict(bytes=16 * n, flops=85 * n * case["iters"])
    if k == "fusion":
        n, hs = case["vw"] * case["vh"] * case["vd"], 8 if case["bins"] <= 8 else 16
        return dict(bytes=4 * case["maps"] * case["w"] * case["h"] + n * (20 + 2 * hs),
                    flops=n * (50 * case["maps"] + case["iters"] * (30 + 8 * case["bins"])))
    n = case["batch"] * case["w"] * case["h"]
    mac = sum(9 * ci * co * (n >> (2 * l)) for (ci, co), l in zip(M.UNET_LAYERS, _UNET_LEVEL))
    npar = sum(9 * ci * co + co for ci, co in M.UNET_LAYERS) + 51
    if not case["train"]:
        return dict(bytes=24 * n + 4 * npar, flops=2 * mac)
    return dict(bytes=24 * n + 28 * npar, flops=6 * mac)


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def _f64(a):
    return torch.as_tensor(np.asarray(a, np.float64) if not torch.is_tensor(a) else a, device=DEV).double()


def _right(a):
    return torch.cat([a[..., 1:], a[..., -1:]], -1)


def _down(a):
    return torch.cat([a[..., 1:, :], a[..., -1:, :]], -2)


def _left(a):
    return torch.cat([a[..., :1], a[..., :-1]], -1)


def _up(a):
    return torch.cat([a[..., :1, :], a[..., :-1, :]], -2)


def _sample(img, xs, ys):
    """Bilinear samples; 0 unless 0 <= floor and floor + 1 <= size - 1."""
    h, w = img.shape
    fx, fy = xs.floor(), ys.floor()
    ok = (fx >= 0) & (fy >= 0) & (fx + 1 <= w - 1) & (fy + 1 <= h - 1)
    i = torch.where(ok, fy * w + fx, torch.zeros_like(fx)).long()
    a, b = xs - fx, ys - fy
    q = img.reshape(-1)
    t1 = a * q[i + 1] + (1 - a) * q[i]
    t2 = a * q[(i + w + 1).clamp(max=h * w - 1)] + (1 - a) * q[(i + w).clamp(max=h * w - 1)]
    return torch.where(ok, b * t2 + (1 - b) * t1, torch.zeros_like(t1))


def _pixels(w, h):
    """1-based pixel coordinates."""
    return (torch.arange(1, w + 1, device=DEV, dtype=torch.float64)[None, :].expand(h, w),
            torch.arange(1, h + 1, device=DEV, dtype=torch.float64)[:, None].expand(h, w))


def _sweep64(ref, srcs, K, rel, planes, win, per_view, ncc_threshold=0.5, zfar=8.0):
    """Per view (best NCC, averaged depth), or (winner's cost, depth, volume)."""
    ref, srcs = _f64(ref), _f64(srcs)
    h, w = ref.shape
    r = win // 2
    invK = np.linalg.inv(K)
    X, Y = _pixels(w, h)

    def mean(a):
        return F.avg_pool2d(F.pad(a[None, None], (r, r, r, r), mode="reflect"), win, 1)[0, 0]

    def std(m, q):
        return (q - m * m).clamp(min=0).sqrt()
    rm = mean(ref)
    rs = std(rm, mean(ref * ref))
    V, P = len(rel), len(planes)
    best = torch.zeros((V, h, w), device=DEV, dtype=torch.float64)
    depth = torch.zeros_like(best)
    vol = None if per_view else torch.zeros((P, h, w), device=DEV, dtype=torch.float64)
    for v, (R, t) in enumerate(rel):
        for p, d in enumerate(planes):
            M3 = np.array(R, np.float64)
            M3[:, 2] += np.asarray(t, np.float64) / float(d)
            H = K @ M3 @ invK
            H = H / H[2, 2]
            z = H[2, 0] * X + H[2, 1] * Y + H[2, 2]
            wi = _sample(srcs[v], (H[0, 0] * X + H[0, 1] * Y + H[0, 2]) / z - 1,
                         (H[1, 0] * X + H[1, 1] * Y + H[1, 2]) / z - 1)
            m = mean(wi)
            s = std(m, mean(wi * wi))
            ncc = torch.where((rs < 1e-4) | (s < 1e-4), torch.zeros_like(m), (mean(ref * wi) - rm * m) / (rs * s))
            if per_view:
                win_ = ncc > best[v]
                best[v] = torch.where(win_, ncc, best[v])
                depth[v] = torch.where(win_, torch.full_like(m, float(d)), depth[v])
            else:
                vol[p] += ncc
    if per_view:
        use = best > ncc_threshold
        cnt = use.sum(0)
        avg = (depth * use).sum(0) / cnt.clamp(min=1)
        return best, torch.where(cnt > 0, avg, torch.full_like(avg, zfar))
    vol = (1 - vol / V).clamp(min=0)
    q = vol.bfloat16()
    lab = q.float().argmin(0)
    return (q.gather(0, lab[None])[0].double(),
            torch.as_tensor(np.asarray(planes, np.float64), device=DEV)[lab], vol)


def _tensor64(ref255, beta=0.0, gamma=1.0):
    r = ref255 / 255
    gx, gy = _right(r) - r, _down(r) - r
    d = (gx * gx + gy * gy).sqrt()
    one = torch.where(d > 0, d, torch.ones_like(d))
    gx, gy = gx / one, gy / one
    k = torch.exp(-beta * d.pow(gamma))
    flat = d <= 0
    return (r, torch.where(flat, torch.ones_like(d), k * gx * gx + gy * gy),
            torch.where(flat, torch.zeros_like(d), (k - 1) * gx * gy),
            torch.where(flat, torch.ones_like(d), k * gy * gy + gx * gx))


def _pq64(p, q, u, vx, vy, T, a0, a1, sigma):
    """The dual steps of the regulariser."""
    t11, t12, t22 = T
    x, y = _right(u) - u - vx, _down(u) - u - vy
    px, py = p[0] + a1 * sigma * (t11 * x + t12 * y), p[1] + a1 * sigma * (t12 * x + t22 * y)
    d = (px * px + py * py).sqrt().clamp(min=1)
    qx, qy = q[0] + a0 * sigma * (_right(vx) - vx), q[1] + a0 * sigma * (_down(vy) - vy)
    qz = q[2] + a0 * sigma * ((_down(vx) - vx) + (_right(vy) - vy)) / 2
    e = (qx * qx + qy * qy + 2 * qz * qz).sqrt().clamp(min=1)
    return (px / d, py / d), (qx / e, qy / e, qz / e)


def _primal64(p, q, T, a0, a1):
    """The regulariser's part of the primal steps of u, vx, vy."""
    t11, t12, t22 = T
    px, py = p
    qx, qy, qz = q
    lx, ux = px - _left(px), px - _up(px)
    ly, uy = py - _left(py), py - _up(py)
    du = t11 * lx + t12 * ly + t12 * ux + t22 * uy
    return (a1 * du, a1 * (t11 * px + t12 * py) + a0 * (qx - _left(qx) + qz - _up(qz)),
            a1 * (t12 * px + t22 * py) + a0 * (qz - _left(qz) + qy - _up(qy)))


def _tgv64(case, s):
    lam, a0, a1, tau, sigma = 0.5, 2.0, 1.5, 0.02, 1.0
    ref01, *T = _tensor64(_f64(s["ref"]))
    h, w = ref01.shape
    X, Y = _pixels(w, h)
    K, invK = s["K"].astype(np.float64).reshape(3, 3), s["invK"].astype(np.float64).reshape(3, 3)
    srcs = _f64(s["srcs"]) / 255
    u = _f64(s["start"]) if case["start"] == "depth" else torch.ones_like(ref01)

    def mul(A, x, y, z):
        return [A[i, 0] * x + A[i, 1] * y + A[i, 2] * z for i in range(3)]
    total = 0
    for _ in range(case["warps"]):
        u0 = u.clone()
        It, Iu = [], []
        for v in range(case["views"]):
            R, t = s["R"][v].astype(np.float64).reshape(3, 3), s["t"][v].astype(np.float64)
            k3 = mul(invK, X, Y, 1.0)
            x3 = [a + float(b) for a, b in zip(mul(R, *[u0 * c for c in k3]), t)]
            q = mul(K, *x3)
            Iw = _sample(srcs[v], q[0] / q[2] - 1, q[1] / q[2] - 1)
            d3 = mul(R @ invK, X, Y, 1.0)
            fx = K[0, 0] * (d3[0] * x3[2] - x3[0] * d3[2]) / (x3[2] * x3[2])
            fy = K[1, 1] * (d3[1] * x3[2] - x3[1] * d3[2]) / (x3[2] * x3[2])
            Iu.append((_right(Iw) - Iw) * fx + (_down(Iw) - Iw) * fy)
            It.append(Iw - ref01)
        It, Iu = torch.stack(It), torch.stack(Iu)
        z = torch.zeros_like(u)
        ub, vx, vy, vxb, vyb, p, q, r = u, z, z, z, z, (z, z), (z, z, z), torch.zeros_like(It)
        hist = []
        for i in range(case["iters"]):
            p, q = _pq64(p, q, ub, vxb, vyb, T, a0, a1, sigma)
            r = (r + sigma * lam * (It + (u - u0) * Iu)).clamp(-1, 1)
            du, dx, dy = _primal64(p, q, T, a0, a1)
            un = u + tau * du - tau * lam * (r * Iu).sum(0)
            xn, yn = vx + tau * dx, vy + tau * dy
            ub, vxb, vyb = 2 * un - u, 2 * xn - vx, 2 * yn - vy
            u, vx, vy = un, xn, yn
            total += 1
            if case["tol"] > 0 and (i + 1) % 10 == 0:
                gx, gy = _right(u) - u - vx, _down(u) - u - vy
                tx, ty = T[0] * gx + T[1] * gy, T[1] * gx + T[2] * gy
                a, b = _right(vx) - vx, _down(vy) - vy
                c = 0.5 * ((_down(vx) - vx) + (_right(vy) - vy))
                E = float((a1 * (tx * tx + ty * ty).sqrt() + a0 * (a * a + b * b + 2 * c * c).sqrt()).sum() +
                          lam * (It + (u - u0) * Iu).abs().sum())
                hist.append(E)
                if len(hist) > 5 and abs(hist[-6] - E) <= case["tol"] * 5 * abs(hist[-6]):
                    break
    return u


def _denoise64(ref255, depth, iters, near=0.4, far=8.0, lam=0.3, tau=0.02, sigma=6.0, theta=1.0):
    _, t11, t12, t22 = _tensor64(_f64(ref255))
    depth = _f64(depth)
    o = (depth - near) / (far - near)
    raw = -(depth - near) * sigma / (far - near)
    r, px, py = torch.zeros_like(o), torch.zeros_like(o), torch.zeros_like(o)
    first = torch.zeros_like(o, dtype=torch.bool)
    first[:, 0] = True
    for it in range(iters):
        c = sigma + 1 if it == 0 else sigma
        x, y = _right(o) - o, _down(o) - o
        px, py = px + c * (t11 * x + t12 * y), py + c * (t12 * x + t22 * y)
        d = (px * px + py * py).sqrt().clamp(min=1)
        px, py = px / d, py / d
        r = (r + raw + sigma * o).clamp(-lam, lam)
        n = o + tau * (torch.where(first, torch.zeros_like(px), px - _left(px)) + py - _up(py)) - tau * r
        o = n + theta * (n - o)
    return o * (far - near) + near


def _sparse64(s, iters, zfar=8.0, a0=2.0, a1=1.5, tau=0.02, sigma=1.0):
    _, *T = _tensor64(_f64(s["ref"]))
    sp = _f64(s["sparse"])
    wgt, ds = (sp > 0).double(), sp / zfar
    u = _f64(s["depth"]) / zfar
    z = torch.zeros_like(u)
    vx, vy, p, q = z, z, (z, z), (z, z, z)
    for _ in range(iters):
        p, q = _pq64(p, q, u, vx, vy, T, a0, a1, sigma)
        du, dx, dy = _primal64(p, q, T, a0, a1)
        u = (u + tau * (du + wgt * ds)) / (1 + tau * wgt)
        vx, vy = vx + tau * dx, vy + tau * dy
    return u * zfar


def _fusion64(case, seed, tau=0.1, lam=0.5, sigma=1.0, thr=0.05):
    depth, Ks, Rs, ts, a, b = _fusion_inputs(case, seed)
    vw, vh, vd, N = case["vw"], case["vh"], case["vd"], case["bins"]
    w, h = case["w"], case["h"]
    a, b = a.astype(np.float64), b.astype(np.float64)
    if N == 2:
        thr = 0.0

    def axis(k, n, shape):
        i = torch.arange(n, device=DEV, dtype=torch.float64)
        return (float(a[k]) + float(b[k] - a[k]) * ((i + 0.5) / n)).reshape(shape)
    x, y, z = axis(0, vw, (1, 1, -1)), axis(1, vh, (1, -1, 1)), axis(2, vd, (-1, 1, 1))
    hist = torch.zeros((N, vd, vh, vw), device=DEV, dtype=torch.int16)
    for m in range(case["maps"]):
        R, t, K = Rs[m].astype(np.float64), ts[m].astype(np.float64), Ks[m].astype(np.float64)
        c = [R[i, 0] * x + R[i, 1] * y + R[i, 2] * z + t[i] for i in range(3)]
        q = [K[i, 0] * c[0] + K[i, 1] * c[1] + K[i, 2] * c[2] for i in range(3)]
        px, py = q[0] / q[2], q[1] / q[2]
        ok = ~((px < 0) | (px > w - 1) | (py < 0) | (py > h - 1))
        px, py = torch.where(ok, px, torch.zeros_like(px)), torch.where(ok, py, torch.zeros_like(py))
        fx, fy = px.floor(), py.floor()
        x0, y0 = fx.long(), fy.long()
        x1, y1 = (x0 + 1).clamp(max=w - 1), (y0 + 1).clamp(max=h - 1)
        d = depth[m].double()
        l0 = d[y0, x0] + (py - fy) * (d[y1, x0] - d[y0, x0])
        l1 = d[y0, x1] + (py - fy) * (d[y1, x1] - d[y0, x1])
        sd = l0 + (px - fx) * (l1 - l0) - q[2]
        mid = torch.zeros_like(sd) if thr == 0 else \
            torch.minimum(torch.floor((sd + thr) / (2 * thr) * (N - 3) + 1 + 0.5), torch.full_like(sd, N - 2))
        bn = torch.where(sd >= thr, torch.full_like(sd, N - 1), torch.where(sd <= -thr, torch.zeros_like(sd), mid))
        bn = torch.where(ok, bn, torch.full_like(bn, -1))
        for k in range(N):
            hist[k] += bn == k
        del c, q, px, py, fx, fy, x0, y0, x1, y1, l0, l1, sd, mid, bn
    cen = [-1.0] + [2.0 * (k - 1) / (N - 3) - 1 if N > 3 else 0.0 for k in range(1, N - 1)] + [1.0]
    W = hist.sum(0, dtype=torch.int32)
    Wj = []
    for k in range(N):
        W = W - 2 * hist[k]
        Wj.append(W.float())
    del hist, W
    u = torch.zeros((vd, vh, vw), device=DEV, dtype=torch.float64)
    v = torch.zeros_like(u)
    p = [torch.zeros_like(u) for _ in range(3)]
    inf = float("inf")

    def back(q, dim):
        o = q.clone()
        o.narrow(dim, 1, q.shape[dim] - 1).sub_(q.narrow(dim, 0, q.shape[dim] - 1))
        return o

    def fwd(q, dim):
        o = torch.zeros_like(q)
        n = q.shape[dim] - 1
        torch.sub(q.narrow(dim, 1, n), q.narrow(dim, 0, n), out=o.narrow(dim, 0, n))
        return o
    for _ in range(case["iters"]):
        uu = u + tau * (back(p[0], 2) + back(p[1], 1) + back(p[2], 0))
        lo = hi = None
        for i in range(N + 1):
            al, bl = cen[i - 1] if i > 0 else -inf, None
            if N - 1 - i >= 0:
                bl = torch.add(uu, Wj[i], alpha=tau * lam).clamp_(min=max(-1.0, al))   # B[N-1-i] is W_{i+1}
            cand = bl if bl is not None else torch.full_like(uu, al)
            lo = cand if lo is None else torch.minimum(lo, cand, out=lo)
            if i > 0:
                bh = torch.add(uu, Wj[i - 1], alpha=tau * lam).clamp_(min=-1.0)   # B[N-i]
                if i < N:
                    bh.clamp_(max=cen[i])
            else:
                bh = torch.full_like(uu, cen[0])
            hi = bh if hi is None else torch.maximum(hi, bh, out=hi)
        new = torch.minimum(torch.maximum(uu.clamp_(min=-1.0), lo), hi)
        v = 2 * new - u
        u = new
        for k, dim in enumerate((2, 1, 0)):
            p[k] = p[k].add_(fwd(v, dim), alpha=sigma)
        d = (p[0] * p[0]).addcmul_(p[1], p[1]).addcmul_(p[2], p[2]).sqrt_().clamp_(min=1)
        for k in range(3):
            p[k].div_(d)
    return dict(u=u.reshape(-1), v=v.reshape(-1), p=torch.stack(p).reshape(3, -1), hist=None)


def _unet64(case, seed):
    s = _unet_inputs(case, seed)
    par = _f64(_unet_params(seed)).requires_grad_(case["train"])
    o = 0
    layers = []
    for ci, co in M.UNET_LAYERS:
        layers.append((par[o:o + 9 * ci * co].reshape(co, ci, 3, 3), par[o + 9 * ci * co:o + 9 * ci * co + co]))
        o += 9 * ci * co + co
    hw, hb = par[o:o + 48].reshape(3, 16, 1, 1), par[o + 48:o + 51]

    def conv(l, a):
        return F.relu(F.conv2d(a, layers[l][0], layers[l][1], padding=1))

    def cat(a, b):
        return torch.cat([F.interpolate(a, scale_factor=2, mode="nearest"), b], 1)
    ds, dsh, clip, us, vs, wu, wv = M.UNET_DEFAULT_NORM
    wta = _f64(s["wta"])
    x = torch.stack([wta * ds + dsh, 1 - _f64(s["cost"]).clamp(0, clip), _f64(s["ref"]) / 255 - 0.5], 1)
    x = F.pad(x, (0, 0, 0, 0, 0, 13))
    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, F.avg_pool2d(e0, 2)))
    e2 = conv(5, conv(4, F.avg_pool2d(e1, 2)))
    e3 = conv(7, conv(6, F.avg_pool2d(e2, 2)))
    d2 = conv(9, conv(8, cat(e3, e2)))
    d1 = conv(11, conv(10, cat(d2, e1)))
    d0 = conv(13, conv(12, cat(d1, e0)))
    out = F.conv2d(d0, hw, hb)
    u, v = wta + us * out[:, 0], vs * out[:, 1:]
    if not case["train"]:
        return dict(u=u, v=v)
    loss = (wu * (u - _f64(s["ut"])) ** 2 + wv * ((v - _f64(s["vt"])) ** 2).sum(1)).mean()
    g, = torch.autograd.grad(loss, par)
    return dict(loss=np.float64(loss.detach().cpu()), grads=g.cpu().numpy())


def exact(case, seed):
    k = case["kind"]
    if k == "sweep":
        fr = _room(seed, case["w"], case["h"], case["views"])
        planes = _planes(case["planes"])
        if case["mode"] == "per_view":
            best, depth = _sweep64(fr.ref, fr.srcs, fr.ref_cam.K_1based, _rel(fr), planes, case["window"], True)
            return dict(depth=depth, labels=None, best=best)
        best, depth, vol = _sweep64(fr.ref, fr.srcs, fr.ref_cam.K_1based, _rel(fr), planes, case["window"], False)
        out = dict(depth=depth, labels=None, best=best)
        return dict(out, cost=vol) if case["w"] * case["h"] % 8 == 0 else out
    if k == "batch":
        out = []
        for f in _batch_frames(case, seed):
            best, depth, _ = _sweep64(f["ref"], f["srcs"], f["K1"], f["rel"], f["depths"].cpu().numpy(), f["window"],
                                      False)
            out.append(dict(depth=depth, labels=None, best=best))
        return out
    if k == "handle":
        fr = _room(seed, case["w"], case["h"], case["views"])
        _, depth = _sweep64(fr.ref, fr.srcs, fr.ref_cam.K_1based, _rel(fr), _planes(case["planes"]), case["window"], True)
        return dict(depth=depth.cpu().numpy(), denoised=_denoise64(fr.ref, depth, case["iters"]).cpu().numpy(), gray=None)
    if k == "fusion":
        return _fusion64(case, seed)
    if k == "unet":
        return _unet64(case, seed)
    s = prepare(case, seed)
    if k == "tgv2":
        return dict(u=_tgv64(case, s), iters=None)
    if k == "denoise":
        return dict(depth=_denoise64(s["ref"], s["start"], case["iters"]))
    return dict(depth=_sparse64(s, case["iters"]))
