"""What the bundle adjuster is timed and compared on.

Each case is one call, or one batch of calls, as a structure-from-motion
program makes it through the public entry points: single adjustments in both
precisions and with both solvers (the smallest local window up to the
2000-camera scene), batches of local windows, camera registration, the
per-camera intrinsics refinement and the plain error of a model. ``prepare``
makes the scene a program has in hand, ``run`` is the call, ``exact`` restates
it in 64-bit torch without this package.
"""
import ctypes
import math

import numpy as np
import torch

from sfmtory_gb300 import abi, native
from sfmtory_gb300.problem import Problem, look_at_pose, perturb_pose

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
MODELS = {"PINHOLE": abi.PINHOLE, "SIMPLE_RADIAL": abi.SIMPLE_RADIAL, "RADIAL": abi.RADIAL, "OPENCV": abi.OPENCV}
LOSSES = {"none": abi.LOSS_NONE, "huber": abi.LOSS_HUBER, "cauchy": abi.LOSS_CAUCHY}
DOF = {abi.PINHOLE: 4, abi.SIMPLE_RADIAL: 4, abi.RADIAL: 5, abi.OPENCV: 8}


def _adjust(name, **kw):
    case = dict(kind="adjust", layout="loop", model="RADIAL", images=100, points=10000, cameras=0, views="poisson",
                outliers=0.0, fixed_intrinsics=False, loss="huber", loss_px=2.0, iterations=50, mixed=False,
                device=False)
    case.update(kw)
    return dict(case, name=name) if name else case


def listed():
    return [
        # The smallest call: the local adjustment after one image was added to
        # a growing reconstruction (one camera, its intrinsics held).
        _adjust("window9_fp64", layout="arc", model="SIMPLE_RADIAL", images=9, points=700, cameras=1,
                fixed_intrinsics=True),
        # A turntable scene: 16 cameras that all see every point, squared loss.
        _adjust("ring16_fp64", layout="arc", model="PINHOLE", images=16, points=2000, views="all", loss="none"),
        # A temple-sized photo set with lens distortion, 5 % of its matches off
        # by some pixels: the few robust iterations between two filter rounds.
        _adjust("opencv47_fp64", model="OPENCV", images=47, points=20000, outliers=0.05, loss_px=1.0, iterations=8),
        # The global adjustment of a video: one camera shared by all images.
        _adjust("video300_fp64", images=300, points=40000, cameras=1),
        # A drone survey, every image its own camera, dense reduced system.
        _adjust("radial500_mixed", model="SIMPLE_RADIAL", images=500, points=200000, views="geometric", loss="none",
                mixed=True),
        # The largest scene: 2000 cameras, six million observations, PCG.
        _adjust("radial2000_mixed", images=2000, points=1000000, views="power", loss="none", mixed=True),
        # A large scene that a program keeps on the GPU, all in 64 bits, PCG.
        _adjust("radial1100_fp64_device", images=1100, points=150000, views="power", loss="none", device=True),
        # Local adjustments of many places of a large reconstruction at once,
        # with free intrinsics and, as growing reconstructions do, held ones.
        dict(name="windows128_mixed", kind="windows", windows=128, scale=0.25, fixed_intrinsics=False, mixed=True),
        dict(name="windows32_fp64", kind="windows", windows=32, scale=0.2, fixed_intrinsics=True, mixed=False),
        # Registration of the next images against the points already there.
        dict(name="pnp512", kind="pnp", images=512, low=200, high=2000, outliers=0.3),
        # Calibration with poses and points held: one camera for all images.
        dict(name="intrinsics1", kind="intrinsics", model="OPENCV", cameras=1, images=47, points=20000),
        # The error of a whole model, printed after each stage.
        dict(name="mean_error", kind="mean_error", model="RADIAL", images=800, points=300000),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["window", "scene", "scene", "video", "large", "windows", "pnp", "intrinsics", "mean_error"])
    if kind == "window":
        return _adjust(None, layout="arc", model=rng.choice(list(MODELS)), images=rng.randint(6, 40),
                       points=_log(rng, 400, 8000), cameras=1, fixed_intrinsics=True,
                       loss=rng.choice(["huber", "cauchy"]), mixed=rng.random() < 0.25)
    if kind == "scene":
        wrong = rng.choice([0.0, 0.05])
        return _adjust(None, model=rng.choice(list(MODELS)), images=_log(rng, 16, 260), points=_log(rng, 4000, 60000),
                       views=rng.choice(["poisson", "geometric"]), loss=rng.choice(list(LOSSES)), outliers=wrong,
                       iterations=8 if wrong else 50, mixed=rng.random() < 0.4)
    if kind == "video":
        return _adjust(None, model=rng.choice(["SIMPLE_RADIAL", "RADIAL", "OPENCV"]), images=_log(rng, 60, 400),
                       points=_log(rng, 8000, 60000), cameras=rng.randint(1, 4), mixed=rng.random() < 0.3)
    if kind == "large":
        mixed = rng.random() < 0.5
        return _adjust(None, images=_log(rng, 700, 1800 if mixed else 1200),
                       points=_log(rng, 60000, 800000 if mixed else 180000), views="power", loss="none", mixed=mixed,
                       device=rng.random() < 0.5)
    if kind == "windows":
        mixed = rng.random() < 0.5
        return dict(kind="windows", windows=_log(rng, 4, 128 if mixed else 32), scale=rng.uniform(0.05, 0.25),
                    fixed_intrinsics=rng.random() < 0.5, mixed=mixed)
    if kind == "pnp":
        low = _log(rng, 50, 400)
        return dict(kind="pnp", images=_log(rng, 1, 600), low=low, high=low * rng.randint(2, 6),
                    outliers=rng.choice([0.1, 0.3, 0.5]))
    if kind == "intrinsics":
        return dict(kind="intrinsics", model=rng.choice(list(MODELS)), cameras=rng.randint(1, 6),
                    images=rng.randint(12, 80), points=_log(rng, 500, 25000))
    return dict(kind="mean_error", model=rng.choice(list(MODELS)), images=_log(rng, 20, 1000),
                points=_log(rng, 2000, 400000))


# ------------------------------------------------------------------- scenes

def _general(model, c):
    """(fx, fy, cx, cy, k1, k2, p1, p2) of parameter rows c [N, 8] of one model."""
    z = torch.zeros_like(c[:, 0])
    if model == abi.PINHOLE:
        cols = [c[:, 0], c[:, 1], c[:, 2], c[:, 3], z, z, z, z]
    elif model == abi.SIMPLE_RADIAL:
        cols = [c[:, 0], c[:, 0], c[:, 1], c[:, 2], c[:, 3], z, z, z]
    elif model == abi.RADIAL:
        cols = [c[:, 0], c[:, 0], c[:, 1], c[:, 2], c[:, 3], c[:, 4], z, z]
    else:
        cols = [c[:, k] for k in range(8)]
    return torch.stack(cols, 1)


def _columns(model):
    """d(general parameters)/d(the model's parameters), [8, 8]."""
    M = torch.zeros(8, 8, dtype=F64, device=DEVICE)
    if model == abi.PINHOLE:
        M[0, 0] = M[1, 1] = M[2, 2] = M[3, 3] = 1
    elif model in (abi.SIMPLE_RADIAL, abi.RADIAL):
        M[0, 0] = M[1, 0] = M[2, 1] = M[3, 2] = M[4, 3] = 1
        if model == abi.RADIAL:
            M[5, 4] = 1
    else:
        M = torch.eye(8, dtype=F64, device=DEVICE)
    return M


def _rotation(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([
        torch.stack([w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (w * y + x * z)], -1),
        torch.stack([2 * (w * z + x * y), w * w - x * x + y * y - z * z, 2 * (y * z - w * x)], -1),
        torch.stack([2 * (x * z - w * y), 2 * (w * x + y * z), w * w - x * x - y * y + z * z], -1)], -2)


def _pixels(g, pc):
    """Pixels of camera-frame points pc under general parameters g."""
    x, y = pc[:, 0] / pc[:, 2], pc[:, 1] / pc[:, 2]
    fx, fy, cx, cy, k1, k2, p1, p2 = g.unbind(1)
    r2 = x * x + y * y
    rad = 1 + k1 * r2 + k2 * r2 * r2
    xd = x * rad + 2 * p1 * x * y + p2 * (r2 + 2 * x * x)
    yd = y * rad + p1 * (r2 + 2 * y * y) + 2 * p2 * x * y
    return torch.stack([fx * xd + cx, fy * yd + cy], 1)


def _unit(t):
    return t / t.norm(dim=1, keepdim=True)


def _scene(case, seed):
    """A Problem with perturbed start values: images on an arc or around a
    loop, looking at a ball of points, each point in a run of neighbouring
    images (one seen by fewer than two stays unobserved); half a pixel of
    noise, keypoints rounded to float32 as detectors store them; the first
    pose fixed and principal points held."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    nI, nP, model = case["images"], case["points"], MODELS[case["model"]]
    arc = case.get("layout", "loop") == "arc"
    radius = 8.0 if arc else 10.0 if nI < 100 else 16.0
    s = np.deg2rad(np.linspace(-30, 30, nI)) if arc else np.linspace(0, 2 * np.pi, nI, endpoint=False)
    r = radius * (1 + 0.04 * np.sin(2 * s + rng.uniform(0, 6)))
    z = radius * 0.08 * np.sin(3 * s + rng.uniform(0, 6)) + rng.uniform(-0.3, 0.3, nI)
    poses_true = look_at_pose(np.stack([r * np.cos(s), r * np.sin(s), z], 1), rng.normal(0, 0.02 * radius, (nI, 3)))
    nC = case.get("cameras", 0) or nI
    cams_true = np.zeros((nC, 8))
    f = rng.uniform(1000, 1400, nC)
    one_f = model in (abi.SIMPLE_RADIAL, abi.RADIAL)
    cams_true[:, 0] = f
    if not one_f:
        cams_true[:, 1] = f * rng.uniform(0.99, 1.01, nC)
    cams_true[:, 1 if one_f else 2], cams_true[:, 2 if one_f else 3] = 800.0, 600.0
    if one_f:
        cams_true[:, 3] = rng.uniform(-0.05, 0.05, nC)
    if model == abi.RADIAL:
        cams_true[:, 4] = rng.uniform(-0.01, 0.01, nC)
    if model == abi.OPENCV:
        cams_true[:, 4], cams_true[:, 5] = rng.uniform(-0.1, 0.1, nC), rng.uniform(-0.02, 0.02, nC)
        cams_true[:, 6:8] = rng.uniform(-1e-3, 1e-3, (nC, 2))
    cam_of_img = (np.arange(nI, dtype=np.int64) * nC // nI).astype(np.int32)

    def dev(a):
        return torch.as_tensor(a, device=DEVICE)

    u = torch.rand(nP, generator=gen, device=DEVICE, dtype=F64)
    pts = _unit(torch.randn(nP, 3, generator=gen, device=DEVICE, dtype=F64)) * (0.38 * radius * u ** (1 / 3))[:, None]
    v = torch.rand(nP, generator=gen, device=DEVICE, dtype=F64)
    views = case.get("views", "poisson")
    if views == "all":
        count = torch.full((nP,), nI, device=DEVICE)
    elif views == "power":  # density ~ m^-2.5 on [2, 200]
        a, b = 2.0 ** -1.5, float(min(200, nI)) ** -1.5
        count = torch.ceil((a + v * (b - a)) ** (-1 / 1.5)).long()
    elif views == "geometric":  # 2 and more, mean 6
        count = 2 + torch.floor(torch.log1p(-v) / math.log(0.8)).long()
    else:
        count = 2 + torch.poisson(torch.full((nP,), 4.0, device=DEVICE, dtype=F64), generator=gen).long()
    count = count.clamp(2, nI)
    start = torch.rand(nP, generator=gen, device=DEVICE, dtype=F64)
    start = torch.floor(start * ((nI - count + 1) if arc else nI)).long()
    pt = torch.repeat_interleave(torch.arange(nP, device=DEVICE), count)
    img = torch.arange(len(pt), device=DEVICE) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
    img = (img + start[pt]) % nI
    R, t = _rotation(dev(poses_true[:, :4])), dev(poses_true[:, 4:])
    pc = torch.einsum("nij,nj->ni", R[img], pts[pt]) + t[img]
    uv = _pixels(_general(model, dev(cams_true))[dev(cam_of_img).long()[img]], pc)
    ok = (pc[:, 2] > 1e-3) & (uv >= 0).all(1) & (uv[:, 0] < 1600) & (uv[:, 1] < 1200)
    keep = torch.bincount(pt[ok], minlength=nP) >= 2
    ok &= keep[pt]
    img, pt, uv = img[ok], pt[ok], uv[ok]
    uv = uv + 0.5 * torch.randn(uv.shape, generator=gen, device=DEVICE, dtype=F64)
    if case.get("outliers"):
        wrong = torch.rand(len(uv), generator=gen, device=DEVICE) < case["outliers"]
        there = uv + 6 * torch.randn(uv.shape, generator=gen, device=DEVICE, dtype=F64)
        uv = torch.where(wrong[:, None], there, uv)
    uv = uv.float().double()
    start_pts = pts + _unit(torch.randn(pts.shape, generator=gen, device=DEVICE, dtype=F64)) * (0.01 * radius)
    delta = np.concatenate([rng.normal(size=(nI, 3)), rng.normal(size=(nI, 3))], 1)
    delta[:, :3] *= np.deg2rad(1.0) / np.linalg.norm(delta[:, :3], axis=1, keepdims=True)
    delta[:, 3:] *= 0.02 * radius / np.linalg.norm(delta[:, 3:], axis=1, keepdims=True)
    delta[0] = 0
    held = bool(case.get("fixed_intrinsics"))
    cams = cams_true.copy()
    if not held:
        cams[:, : 1 if one_f else 2] *= 1 + 0.03 * rng.choice([-1.0, 1.0], nC)[:, None]
    mask = np.zeros((nC, 8), bool)
    mask[:, 1 if one_f else 2: 3 if one_f else 4] = True
    fixed = np.zeros(nI, bool)
    fixed[0] = True
    return Problem(camera_of_image=cam_of_img, camera_model=np.full(nC, model, np.int32), camera_params=cams,
                   poses=perturb_pose(poses_true, delta), points=start_pts.cpu().numpy(),
                   obs_image=img.int().cpu().numpy(), obs_point=pt.int().cpu().numpy(), obs_xy=uv.cpu().numpy(),
                   fixed_poses=fixed, fixed_cameras=np.full(nC, held), fixed_camera_params=mask)


def _pnp_scene(case, seed):
    """Per image: points four to twelve units away in a 60 degree cone, half
    a pixel of noise at a focal length of 1200, a share of wrong matches."""
    rng = np.random.default_rng(seed)
    Xs, uvs = [], []
    for n in np.random.default_rng(case["images"]).integers(case["low"], case["high"] + 1, case["images"]):
        ax = rng.normal(size=3)
        ax *= rng.uniform(0, 0.5) / np.linalg.norm(ax)
        K = np.array([[0, -ax[2], ax[1]], [ax[2], 0, -ax[0]], [-ax[1], ax[0], 0]])
        th = np.linalg.norm(ax)
        R = np.eye(3) + np.sin(th) / th * K + (1 - np.cos(th)) / th ** 2 * K @ K
        d, xy = rng.uniform(4, 12, n), rng.uniform(-0.55, 0.55, (n, 2))
        pc = np.concatenate([xy * d[:, None], d[:, None]], 1)
        uv = xy + rng.normal(0, 0.5 / 1200, (n, 2))
        wrong = rng.choice(n, int(round(case["outliers"] * n)), replace=False)
        uv[wrong] = rng.uniform(-0.6, 0.6, (len(wrong), 2))
        Xs.append((pc - rng.uniform(-2, 2, 3)) @ R)
        uvs.append(uv)
    return Xs, uvs


def _window_sizes(case):
    """(images, points, model) of each window: 8 to 64 images and, times the
    scale, 500 to 20000 points."""
    rng = np.random.default_rng(case["windows"])
    return [(int(rng.integers(8, 65)), max(20, int(rng.integers(500, 20001) * case["scale"])),
             rng.choice(["PINHOLE", "SIMPLE_RADIAL", "OPENCV"])) for _ in range(case["windows"])]


def _windows(case, seed):
    return [_scene(dict(layout="arc", images=i, points=p, model=str(m), fixed_intrinsics=case["fixed_intrinsics"]),
                   seed * 1000 + k) for k, (i, p, m) in enumerate(_window_sizes(case))]


def _options(case):
    return dict(robust_loss=LOSSES[case.get("loss", "huber")], loss_scale_px=case.get("loss_px", 2.0),
                max_iterations=case.get("iterations", 50),
                precision=abi.PRECISION_MIXED if case.get("mixed") else abi.PRECISION_FP64)


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    kind = case["kind"]
    if kind == "pnp":
        return {"kind": kind, "in": _pnp_scene(case, seed)}
    if kind == "windows":
        return {"kind": kind, "in": _windows(case, seed), "options": _options(case)}
    p = _scene(case, seed)
    if not case.get("device"):
        return {"kind": kind, "in": p, "options": _options(case)}
    pk = abi.PackedProblem(p)
    names = ("camera_of_image", "camera_model", "camera_params", "poses", "points", "obs_image", "obs_point",
             "obs_xy", "fixed_poses", "fixed_cameras", "fixed_camera_params")
    tensors = {k: torch.from_numpy(getattr(pk, k)).to(DEVICE) for k in names}
    struct = abi.SfmbaProblem()
    for k in ("num_images", "num_cameras", "num_points", "num_observations"):
        setattr(struct, k, getattr(pk.struct, k))
    for k, t in tensors.items():
        setattr(struct, k, t.data_ptr())
    out = {k: torch.zeros_like(tensors[k]) for k in ("poses", "points", "camera_params")}
    result = abi.SfmbaResult()
    for k, t in out.items():
        setattr(result, k, t.data_ptr())
    return {"kind": "device", "in": tensors, "struct": struct, "out": out, "result": result,
            "options": abi.default_options(**_options(case))}


def _outputs(r):
    return {"poses": r.poses, "points": r.points, "camera_params": r.camera_params, "initial_cost": r.initial_cost,
            "final_cost": r.final_cost, "iterations": int(r.iterations_run)}


def run(state):
    kind = state["kind"]
    if kind == "adjust":
        return _outputs(native.bundle_adjust_arrays(state["in"], **state["options"]))
    if kind == "device":
        res = state["result"]
        status = native.load().sfmba_bundle_adjust_device(ctypes.byref(state["struct"]),
                                                          ctypes.byref(state["options"]), ctypes.byref(res), None)
        if status != 0:
            raise native.SfmbaError(status, native.load().sfmba_last_error().decode())
        return {**state["out"], "initial_cost": res.initial_cost, "final_cost": res.final_cost,
                "iterations": int(res.iterations_run)}
    if kind == "windows":
        rs = native.bundle_adjust_batched_arrays(state["in"], **state["options"])
        return {"poses": np.concatenate([r.poses for r in rs]), "points": np.concatenate([r.points for r in rs]),
                "camera_params": np.concatenate([r.camera_params for r in rs]),
                "initial_cost": np.array([r.initial_cost for r in rs]),
                "final_cost": np.array([r.final_cost for r in rs]),
                "iterations": np.array([r.iterations_run for r in rs])}
    if kind == "pnp":
        got = native.pnp_ransac_batched(*state["in"], 8.0 / 1200, 2000)
        none = (np.full(7, np.nan), np.zeros(0, bool), 0)
        got = [none if g is None else g for g in got]
        return {"poses": np.stack([g[0] for g in got]), "inliers": np.concatenate([g[1] for g in got]),
                "iterations": np.array([g[2] for g in got])}
    if kind == "intrinsics":
        return {"camera_params": native.refine_intrinsics_arrays(state["in"])}
    return {"mean_error": native.mean_reprojection_error_arrays(state["in"])}


def work(case):
    kind = case["kind"]
    if kind == "pnp":
        n = case["images"] * (case["low"] + case["high"]) / 2
        # 50 hypotheses scored, a DLT over the inliers, twenty pose steps
        return {"bytes": n * (5 * 8 + 1), "flops": n * (50 * 30 + 2 * 12 * 12 + 20 * 120)}
    if kind == "windows":
        sizes = _window_sizes(case)
        images, points = sum(s[0] for s in sizes), sum(s[1] for s in sizes)
        obs, pairs, iters = 6 * points, 21 * points, 8
        D = 6 if case["fixed_intrinsics"] else 12
        factor = sum((s[0] * D) ** 3 / 3 for s in sizes)
    else:
        images, points = case["images"], case["points"]
        track = {"all": case["images"], "power": 5.9, "geometric": 6.0}.get(case.get("views", "poisson"), 6.0)
        obs = points * track
        D = 6 if case.get("fixed_intrinsics") else 6 + DOF[MODELS[case["model"]]]
        n = images * 6 + (0 if case.get("fixed_intrinsics") else (case.get("cameras", 0) or images) * (D - 6))
        pairs = points * track * (track + 1) / 2
        iters = min(8, case.get("iterations", 50))
        factor = n ** 3 / 3
        if case["kind"] == "mean_error":
            return {"bytes": obs * 24 + points * 24 + images * 56, "flops": obs * 60}
        if case["kind"] == "intrinsics":
            return {"bytes": obs * 24 + points * 24 + images * 56, "flops": 8 * obs * (60 * 18 + 2 * 44)}
    data = obs * 24 + points * 48 + images * 240
    if kind == "adjust" and n > 6000:  # matrix-free: twelve products per step
        return {"bytes": data, "flops": iters * obs * (400 + 2 * D * D + 12 * 2 * 4 * (D + 3))}
    return {"bytes": data, "flops": iters * (obs * (400 + 2 * D * D) + pairs * 2 * 3 * D * D + factor)}


# ------------------------------------------------- the same calls in 64 bits

class _Exact:
    """One problem's tensors, its residuals and its Levenberg-Marquardt loop."""

    def __init__(self, p, loss, loss_px):
        def dev(a, dtype):
            return torch.as_tensor(np.asarray(a), device=DEVICE).to(dtype)

        self.loss, self.s = loss, max(loss_px, 1e-9)
        self.img, self.pt, self.xy = dev(p.obs_image, torch.long), dev(p.obs_point, torch.long), dev(p.obs_xy, F64)
        self.cam_of_img = dev(p.camera_of_image, torch.long)
        self.cam = self.cam_of_img[self.img]
        self.model = [int(m) for m in p.camera_model]
        self.maps = torch.stack([_columns(m) for m in self.model])
        self.poses, self.points, self.cams = dev(p.poses, F64), dev(p.points, F64), dev(p.camera_params, F64)
        nI, nC = len(self.poses), len(self.cams)
        slot, n = np.full((nI, 14), -1), 0
        for i in range(nI):
            if not p.fixed_poses[i]:
                slot[i, :6] = range(n, n + 6)
                n += 6
        held = np.zeros(nC, bool) if p.fixed_cameras is None else p.fixed_cameras
        cslot, masked = np.full((nC, 8), -1), []
        for c in range(nC):
            if not held[c]:
                k = DOF[self.model[c]]
                cslot[c, :k] = range(n, n + k)
                masked += [n + q for q in range(k) if p.fixed_camera_params[c][q]]
                n += k
        slot[:, 6:] = cslot[np.asarray(p.camera_of_image)]
        self.n, self.cslot = n, dev(cslot, torch.long)
        self.slot = dev(slot, torch.long)
        self.slot[self.slot < 0] = n  # a spare row and column takes what is held
        self.cslot[self.cslot < 0] = n
        self.masked = dev(np.array(masked, int), torch.long)

    def general(self, cams):
        return torch.einsum("cgm,cm->cg", self.maps, cams)

    def camera_frame(self, poses, points):
        return torch.einsum("nij,nj->ni", _rotation(poses[:, :4])[self.img], points[self.pt]) + poses[self.img, 4:]

    def residual(self, poses, points, cams):
        pc = self.camera_frame(poses, points)
        ok = pc[:, 2] > 1e-9
        pc = torch.where(ok[:, None], pc, torch.ones_like(pc))
        r = _pixels(self.general(cams)[self.cam], pc) - self.xy
        return torch.where(ok[:, None], r, torch.zeros_like(r)), ok, pc

    def weight(self, n):
        if self.loss == "huber":
            return torch.where(n <= self.s, torch.ones_like(n), self.s / n.clamp_min(1e-300))
        if self.loss == "cauchy":
            return 1 / (1 + (n / self.s) ** 2)
        return torch.ones_like(n)

    def cost(self, poses, points, cams):
        n = self.residual(poses, points, cams)[0].norm(dim=1)
        return float((self.weight(n) * n * n).sum())

    def jacobians(self):
        r, ok, pc = self.residual(self.poses, self.points, self.cams)
        iz = 1 / pc[:, 2]
        x, y = pc[:, 0] * iz, pc[:, 1] * iz
        fx, fy, _, _, k1, k2, p1, p2 = self.general(self.cams)[self.cam].unbind(1)
        r2 = x * x + y * y
        rad, kr = 1 + k1 * r2 + k2 * r2 * r2, k1 + 2 * k2 * r2
        dxy = 2 * kr * x * y + 2 * p1 * x + 2 * p2 * y
        dxx = rad + 2 * kr * x * x + 2 * p1 * y + 6 * p2 * x
        dyy = rad + 2 * kr * y * y + 6 * p1 * y + 2 * p2 * x
        A = torch.stack([torch.stack([fx * dxx, fx * dxy], 1), torch.stack([fy * dxy, fy * dyy], 1)], 1)
        z, one = torch.zeros_like(x), torch.ones_like(x)
        dn = torch.stack([torch.stack([iz, z, -x * iz], 1), torch.stack([z, iz, -y * iz], 1)], 1)
        d = A @ dn
        Jx = d @ _rotation(self.poses[:, :4])[self.img]
        q = pc - self.poses[self.img, 4:]
        Jw = torch.cross(q[:, None, :].expand_as(d), d, dim=2)
        gu = torch.stack([x * rad + 2 * p1 * x * y + p2 * (r2 + 2 * x * x), z, one, z, fx * x * r2, fx * x * r2 * r2,
                          fx * 2 * x * y, fx * (r2 + 2 * x * x)], 1)
        gv = torch.stack([z, y * rad + p1 * (r2 + 2 * y * y) + 2 * p2 * x * y, z, one, fy * y * r2, fy * y * r2 * r2,
                          fy * (r2 + 2 * y * y), fy * 2 * x * y], 1)
        Jc = torch.stack([gu, gv], 1) @ self.maps[self.cam]
        w = torch.where(ok, self.weight(r.norm(dim=1)), torch.zeros_like(x))
        return r, w, torch.cat([Jw, d, Jc], 2), Jx

    def pairs(self):
        """Ordered pairs of observations of the same point, a chunk at a time."""
        order = torch.argsort(self.pt, stable=True)
        count = torch.bincount(self.pt, minlength=len(self.points))
        first = torch.cumsum(count, 0) - count
        m = count[self.pt[order]]  # partners of each observation, in point order
        ends = torch.cumsum(m, 0)
        cuts = [0]
        while cuts[-1] < len(order):
            base = int(ends[cuts[-1] - 1]) if cuts[-1] else 0
            cuts.append(max(cuts[-1] + 1, int(torch.searchsorted(ends, base + 500000, right=True))))
        for a, b in zip(cuts[:-1], cuts[1:]):
            mm = m[a:b]
            left = torch.repeat_interleave(torch.arange(a, min(b, len(order)), device=DEVICE), mm)
            off = torch.arange(len(left), device=DEVICE) - torch.repeat_interleave(torch.cumsum(mm, 0) - mm, mm)
            yield order[left], order[first[self.pt[order[left]]] + off]

    def adjust(self, iterations):
        n, N = self.n, self.n + 1
        cost = initial = self.cost(self.poses, self.points, self.cams)
        lam, nu, ran = 1e-3, 2.0, 0
        pairs = list(self.pairs()) if len(self.pt) < 2_000_000 else None
        while ran < iterations and n:
            ran += 1
            before = cost
            r, w, J, Jx = self.jacobians()
            slots = self.slot[self.img]
            WJ = J * w[:, None, None]
            B = torch.zeros(len(self.poses), 14, 14, dtype=F64, device=DEVICE)
            B.index_add_(0, self.img, WJ.transpose(1, 2) @ J)
            b = torch.zeros(N, dtype=F64, device=DEVICE)
            b.index_add_(0, slots.reshape(-1), torch.einsum("nij,ni->nj", WJ, r).reshape(-1))
            E = WJ.transpose(1, 2) @ Jx
            C = torch.zeros(len(self.points), 3, 3, dtype=F64, device=DEVICE)
            C.index_add_(0, self.pt, (Jx * w[:, None, None]).transpose(1, 2) @ Jx)
            g = torch.zeros(len(self.points), 3, dtype=F64, device=DEVICE)
            g.index_add_(0, self.pt, torch.einsum("nij,ni->nj", Jx * w[:, None, None], r))
            base = torch.zeros(N * N, dtype=F64, device=DEVICE)
            base.index_add_(0, (self.slot[:, :, None] * N + self.slot[:, None, :]).reshape(-1), B.reshape(-1))
            base = base.view(N, N)
            diag = base.diagonal().clone()
            taken = False
            for _ in range(8):
                Cd = C + torch.diag_embed(C.diagonal(dim1=1, dim2=2) * lam)
                good = torch.linalg.det(Cd) != 0
                Ci = torch.linalg.inv(torch.where(good[:, None, None], Cd, torch.eye(3, dtype=F64, device=DEVICE)))
                Ci = Ci * good[:, None, None]
                S = base.clone().view(-1)
                EC = E @ Ci[self.pt]
                for a, c in pairs if pairs is not None else self.pairs():
                    at = slots[a][:, :, None] * N + slots[c][:, None, :]
                    S.index_add_(0, at.reshape(-1), -(EC[a] @ E[c].transpose(1, 2)).reshape(-1))
                S = S.view(N, N)[:n, :n]
                S = 0.5 * (S + S.T) + torch.diag(diag[:n] * lam)
                rhs = -b
                rhs = rhs.index_add(0, slots.reshape(-1), torch.einsum("nij,nj->ni", EC, g[self.pt]).reshape(-1))[:n]
                S[self.masked, :] = 0
                S[:, self.masked] = 0
                S[self.masked, self.masked] = 1
                rhs[self.masked] = 0
                L, info = torch.linalg.cholesky_ex(S)
                delta = torch.cholesky_solve(rhs[:, None], L)[:, 0] if int(info) == 0 else torch.linalg.solve(S, rhs)
                delta = torch.cat([delta, delta.new_zeros(1)])
                acc = g.index_add(0, self.pt, torch.einsum("nij,ni->nj", E, delta[slots]))
                points = self.points - torch.einsum("nij,nj->ni", Ci, acc)
                d = delta[self.slot[:, :6]]
                th = d[:, :3].norm(dim=1, keepdim=True)
                half = torch.where(th > 0, torch.sin(0.5 * th) / th.clamp_min(1e-300), torch.full_like(th, 0.5))
                aw, av = torch.cos(0.5 * th), d[:, :3] * half
                bw, bv = self.poses[:, :1], self.poses[:, 1:4]
                poses = torch.cat([aw * bw - (av * bv).sum(1, keepdim=True),
                                   aw * bv + bw * av + torch.cross(av, bv, dim=1), self.poses[:, 4:] + d[:, 3:]], 1)
                cams = self.cams + delta[self.cslot]
                trial = self.cost(poses, points, cams)
                if math.isfinite(trial) and trial < cost:
                    self.poses, self.points, self.cams, cost, taken = poses, points, cams, trial, True
                    lam, nu = max(lam / 3, 1e-12), 2.0
                    break
                lam, nu = lam * nu, nu * 2
            if not taken or (before - cost) / max(before, 1e-12) < 1e-6:
                break
        return {"poses": self.poses, "points": self.points, "camera_params": self.cams, "initial_cost": initial,
                "final_cost": cost, "iterations": ran}

    def refine_intrinsics(self):
        """Each camera's parameters with poses and points held (central
        differences, 30 iterations, Huber at two pixels)."""
        out = self.cams.clone()
        pc_all = self.camera_frame(self.poses, self.points)
        for c in range(len(self.cams)):
            mine = (self.cam == c) & (pc_all[:, 2] > 1e-9)
            if int((self.cam == c).sum()) < 8:
                continue
            pc, xy, k = pc_all[mine], self.xy[mine], DOF[self.model[c]]

            def res(v):
                return _pixels((self.maps[c] @ v)[None].expand(len(pc), 8), pc) - xy

            def total(v):
                m = res(v).norm(dim=1)
                return float((self.weight(m) * m * m).sum())

            cur, lam = out[c].clone(), 1e-3
            cost = total(cur)
            for _ in range(30):
                r = res(cur)
                w = self.weight(r.norm(dim=1))[:, None]
                J = []
                for q in range(k):
                    up, down = cur.clone(), cur.clone()
                    up[q] += 1e-6
                    down[q] -= 1e-6
                    J.append((res(up) - res(down)) / 2e-6)
                J = torch.stack(J, 2)
                H = torch.einsum("nia,nib->ab", J * w[:, :, None], J)
                gr = torch.einsum("nia,ni->a", J * w[:, :, None], r)
                taken = False
                for _ in range(8):
                    d = torch.linalg.solve(H + torch.diag(lam * H.diagonal().clamp_min(1e-12)), -gr)
                    new = cur.clone()
                    new[:k] += d
                    trial = total(new)
                    if math.isfinite(trial) and trial < cost:
                        cur, cost, lam, taken = new, trial, max(lam / 3, 1e-12), True
                        break
                    lam *= 3
                if not taken:
                    break
            out[c] = cur
        return {"camera_params": out}


def exact(case, seed):
    kind = case["kind"]
    if kind == "pnp":
        return None  # a pose that depends on which random samples were drawn
    if kind == "windows":
        got = [_Exact(p, case.get("loss", "huber"), 2.0).adjust(50) for p in _windows(case, seed)]
        cat = {k: torch.cat([g[k] for g in got]) for k in ("poses", "points", "camera_params")}
        one = {k: np.array([g[k] for g in got]) for k in ("initial_cost", "final_cost", "iterations")}
        return {**cat, **one}
    e = _Exact(_scene(case, seed), case.get("loss", "huber"), case.get("loss_px", 2.0))
    if kind == "intrinsics":
        return e.refine_intrinsics()
    if kind == "mean_error":
        r, ok, _ = e.residual(e.poses, e.points, e.cams)
        return {"mean_error": float(r.norm(dim=1).sum() / ok.sum())}
    if e.n > 6000:
        return None  # solved inexactly by design: no step has one right value
    return e.adjust(case["iterations"])
