"""Workloads of the registration core, each through the entry point that a user's program calls.

``listed`` holds one case per use, ``draw`` further sizes of the same ranges, ``prepare`` what the
program has in hand before the call, ``run`` the call, ``work`` the bytes and operations that the
call cannot do without, and ``exact`` its result from plain torch in 64 bits.

The scenes are those of the package's generator (rooms, textured stereo views, ring-sensor scans
of a street), sampled on the GPU because the inputs are made many times.
"""
import math

import numpy as np
import torch

from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path
from rkhs_ba_gb300 import scenes
from rkhs_ba_gb300.proposal import ProposalNet, ScenePool

D = torch.float64
PARAMS = {"room": "geometric", "color": "color", "lidar": "lidar_semantic"}
RECORD = {"room": 16, "color": 16 + 32, "lidar": 16 + 16 + 80}   # bytes of one packed point


def listed():
    return [
        # a single similarity query between two small host clouds: latency and launches
        {"name": "ip_room_1k", "kind": "ip", "scene": "room", "n": 1000, "ell": 0.25},
        # place recognition: one view pair scored at the 24 rotations of a start grid
        {"name": "cos_grid_color_50k", "kind": "cos", "scene": "color", "n": 50000, "ell": 0.4, "poses": 24},
        # tracking small colour frames from host memory: a whole registration from a motion prior
        {"name": "align_color_4k_host", "kind": "align_host", "scene": "color", "n": 4001, "ell": 0.4, "iters": 60},
        # stereo odometry: the configured colour pair at the configured lengthscale, clouds resident
        {"name": "align_color_50k", "kind": "align", "scene": "color", "n": 50000, "ell": 1.0, "iters": 60},
        # indoor scans without colour, a few iterations for each sweep
        {"name": "align_room_10k", "kind": "align", "scene": "room", "n": 10000, "ell": 0.25, "iters": 6},
        # semantic LiDAR odometry at the sensor's full resolution, a few iterations for each sweep
        {"name": "align_lidar_128k", "kind": "align", "scene": "lidar", "n": 128000, "ell": 0.2, "iters": 5},
        # refinement of global-registration hypotheses: several uneven pairs in one batch
        {"name": "align_batch_8", "kind": "align_batch", "scene": "color", "n": 50000, "ell": 0.4, "iters": 60, "pairs": 8},
        # correspondences for a mapping back end, on the host as CSR
        {"name": "assoc_color_30k", "kind": "assoc", "scene": "color", "n": 30011, "ell": 0.4, "cap": 32},
        # the same with a non-isotropic geometric kernel
        {"name": "aniso_color_20k", "kind": "aniso", "scene": "color", "n": 20000, "cap": 64},
        # an RGB-D frame to a registration-ready cloud and back to the host
        {"name": "rgbd_50k", "kind": "rgbd", "rows": 370, "cols": 1226, "n": 50000},
        # bundle adjustment of a window of keyframes, every pair an edge
        {"name": "window_8", "kind": "window", "scene": "color", "frames": 8, "lo": 20000, "hi": 60000, "outer": 6},
        # one optimisation step of the pose-proposal network
        {"name": "train_64", "kind": "train", "pairs": 64, "points": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    kind = rng.choice(["ip", "ip", "cos", "align_host", "align", "align", "align", "align_batch", "assoc", "aniso", "rgbd",
                       "window", "train"])
    scene = rng.choice(["room", "color", "lidar"])
    c = {"kind": kind}
    if kind in ("ip", "assoc"):
        c.update(scene=scene, n=_log(rng, 500, 30000), ell=round(rng.uniform(0.1, 0.5), 3))
        if kind == "assoc":
            c["cap"] = rng.randint(8, 48)
    elif kind == "cos":
        c.update(scene=rng.choice(["room", "color"]), n=_log(rng, 1000, 40000), ell=round(rng.uniform(0.2, 0.5), 3),
                 poses=rng.choice([8, 24, 60]))
        c["poses"] = min(c["poses"], max(8, 24 * 50000 // c["n"] // 8 * 8))
    elif kind in ("align", "align_host"):
        # without colour the path of the poses is ill-conditioned: a few iterations, so that results can be compared
        most = {"room": 20000, "color": 45000, "lidar": 100000}[scene] if kind == "align" else 8000
        c.update(scene=scene, n=_log(rng, 1000, most), ell=round(rng.uniform(0.15, 0.6), 3),
                 iters=rng.randint(8, 40) if scene == "color" else rng.randint(2, 5))
    elif kind == "align_batch":
        c.update(scene="color", n=_log(rng, 3000, 40000), ell=round(rng.uniform(0.2, 0.4), 3), iters=rng.randint(12, 40),
                 pairs=rng.randint(2, 8))
    elif kind == "aniso":
        c.update(scene="color", n=_log(rng, 1000, 18000), cap=rng.randint(16, 64))
    elif kind == "rgbd":
        c.update(rows=rng.choice([240, 370, 480]), cols=rng.choice([320, 640, 1226]), n=_log(rng, 2000, 45000))
    elif kind == "window":
        lo = _log(rng, 3000, 15000)
        c.update(scene="color", frames=rng.randint(3, 6), lo=lo, hi=3 * lo, outer=rng.randint(2, 4))
    else:
        c.update(pairs=rng.randint(8, 60), points=rng.choice([256, 384, 512]))
    return c


# ------------------------------------------------------------------ scenes
def _gen(seed, k):
    return torch.Generator("cuda").manual_seed((int(seed) * 7919 + 101 * k) % (2 ** 62))


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=D, device="cuda")


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=D)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=D)


def _move(T, p):
    T = _t(T)
    return p @ T[:3, :3].T + T[:3, 3]


def _room(spheres, n, g):
    """n points, uniform by area, of a 20 x 20 x 5 m room with three spheres."""
    areas = _t([400.0, 400.0] + [100.0] * 4 + [4 * math.pi * r * r for _, r in spheres])
    which = torch.multinomial(areas, n, replacement=True, generator=g)
    u, v, h = _uniform(g, n, -10, 10), _uniform(g, n, -10, 10), _uniform(g, n, 0, 5)
    d = _normal(g, n, 3)
    d = d / d.norm(dim=1, keepdim=True)
    full = lambda x: torch.full_like(u, x)  # noqa: E731
    faces = [(u, v, full(0)), (u, v, full(5)), (full(-10), v, h), (full(10), v, h), (u, full(-10), h), (u, full(10), h)]
    p = torch.zeros(n, 3, device="cuda", dtype=D)
    for k, f in enumerate(faces):
        p = torch.where((which == k)[:, None], torch.stack(f, 1), p)
    for k, (c, r) in enumerate(spheres):
        p = torch.where((which == 6 + k)[:, None], _t(c) + r * d, p)
    return p


def _raycast(world, o, d):
    best = torch.full((d.shape[0],), math.inf, device="cuda", dtype=D)
    for c, nrm, ax, hw, hh in world.patches:
        c, nrm, ax = _t(c), _t(nrm), _t(ax)
        s = ((c - o) @ nrm) / (d @ nrm)
        ok = (s > 0.1) & torch.isfinite(s) & (s < best)
        if hw < 1e8:
            q = o + s[:, None] * d - c
            ok &= ((q @ ax).abs() <= hw) & ((q @ torch.linalg.cross(nrm, ax)).abs() <= hh)
        best = torch.where(ok, s, best)
    hit = torch.isfinite(best) & (best < 80.0)
    return o + torch.where(hit, best, 0.0)[:, None] * d, hit


def _texture(world, p):
    f, ph, am = _t(world.freq), _t(world.phase), _t(world.amp)
    return torch.stack([0.5 + 0.5 * torch.tanh(1.2 * (am[c] * torch.sin(p @ f[c].T + ph[c])).sum(1)) for c in range(3)], 1)


def _view(world, cam, n, g):
    """The n pixels of highest gradient of a pinhole view: camera-frame points, 5 features."""
    u, v = _uniform(g, 4 * n, 0, 1226), _uniform(g, 4 * n, 0, 370)
    T = _t(cam)

    def cast(uu, vv):
        d = torch.stack([(uu - 613.0) / 718.0, (vv - 185.0) / 718.0, torch.ones_like(uu)], 1)
        d = d / d.norm(dim=1, keepdim=True)
        return _raycast(world, T[:3, 3], d @ T[:3, :3].T)

    pw, ok = cast(u, v)
    pu, ku = cast(u + 1.0, v)
    pv, kv = cast(u, v + 1.0)
    col = _texture(world, pw)
    grey = col.mean(1) * 255.0
    gx, gy = _texture(world, pu).mean(1) * 255.0 - grey, _texture(world, pv).mean(1) * 255.0 - grey
    mag = torch.where(ok & ku & kv, torch.hypot(gx, gy), torch.full_like(gx, -1.0))
    keep = torch.sort(torch.argsort(mag, descending=True, stable=True)[:n]).values
    pc = (pw[keep] - T[:3, 3]) @ T[:3, :3]
    feat = torch.cat([col[keep], torch.stack([gx[keep], gy[keep]], 1) / 500.0 + 0.5], 1)
    return pc, feat.clamp(0, 1)


def _scan(boxes, poles, S, n, g):
    """A 64-beam ring scan of a street: points, intensity and 19-class label distributions."""
    el = torch.deg2rad(torch.linspace(-25.0, 3.0, 64, device="cuda", dtype=D))
    az = torch.linspace(-math.pi, math.pi, 2049, device="cuda", dtype=D)[:-1]
    E, A = torch.meshgrid(el, az, indexing="ij")
    d = torch.stack([E.cos() * A.cos(), E.cos() * A.sin(), E.sin()], -1).reshape(-1, 3) @ _t(S)[:3, :3].T
    o = _t(S)[:3, 3]
    s = (-1.8 - o[2]) / d[:, 2]
    best = torch.where((s > 0) & torch.isfinite(s), s, torch.full_like(s, math.inf))
    lab = torch.zeros(d.shape[0], dtype=torch.int64, device="cuda")

    def take(ok, s, label):
        nonlocal best, lab
        best = torch.where(ok, s, best)
        lab = torch.where(ok, torch.full_like(lab, label), lab)

    for lo, hi in boxes:
        t1, t2 = (_t(lo) - o) / d, (_t(hi) - o) / d
        tn, tf = torch.minimum(t1, t2).amax(1), torch.maximum(t1, t2).amin(1)
        take((tn <= tf) & (tn > 0) & (tn < best), tn, 2)
    for c, r in poles:
        oc = o[:2] - _t(c)
        a, b, cc = (d[:, :2] ** 2).sum(1), 2 * (d[:, :2] @ oc), float((oc ** 2).sum()) - r * r
        disc = b * b - 4 * a * cc
        s = (-b - disc.clamp(min=0).sqrt()) / (2 * a)
        take((disc > 0) & (s > 0) & (s < best) & (o[2] + s * d[:, 2] < 6.0), s, 5)
    hit = (torch.isfinite(best) & (best > 2.0) & (best < 80.0)).nonzero()[:, 0]
    if len(hit) > n:
        hit = hit[torch.sort(torch.randperm(len(hit), generator=g, device="cuda")[:n]).values]
    pw, lab = o + best[hit, None] * d[hit], lab[hit]
    pc = (pw - o) @ _t(S)[:3, :3] + 0.01 * _normal(g, len(hit), 3)
    inten = (0.3 + 0.1 * lab + 0.2 * torch.sin(0.7 * pw[:, 0]) * torch.cos(0.5 * pw[:, 1])).clamp(0, 1)
    logits = _normal(g, len(hit), 19)
    logits[torch.arange(len(hit), device="cuda"), lab] += 4.0
    return pc, inten[:, None], torch.softmax(logits, 1)


def _cloud(xyz, feat=None, lab=None):
    h = lambda a: None if a is None else a.to(torch.float32).cpu().numpy()  # noqa: E731
    return CvoPointCloud(h(xyz), h(feat), h(lab))


def _unit(rng):
    d = rng.normal(size=3)
    return d / np.linalg.norm(d)


def _pair(scene, n, seed):
    """(source, target, T) with source ~= T target."""
    rng = np.random.default_rng(seed)
    if scene == "room":
        sph = scenes._room_surfaces(rng)
        G = scenes.make_T(scenes.random_rotation(rng, math.radians(10)), _unit(rng) * rng.uniform(0, 0.5))
        tgt = _move(G, _room(sph, n, _gen(seed, 2))) + 0.01 * _normal(_gen(seed, 3), n, 3)
        return _cloud(_room(sph, n, _gen(seed, 1))), _cloud(tgt), scenes.inv_T(G)
    if scene == "color":
        w = scenes._TexturedWorld(rng)
        cam = scenes.make_T(scenes.rot_axis_angle([0, 1, 0], math.radians(rng.uniform(-3, 3))), [0, 0, rng.uniform(0.5, 1.5)])
        return _cloud(*_view(w, np.eye(4), n, _gen(seed, 1))), _cloud(*_view(w, cam, n, _gen(seed, 2))), cam
    boxes, poles = scenes._street(rng)
    S = scenes.make_T(scenes.random_rotation(rng, math.radians(5)), _unit(rng) * [1, 1, 0.1] * rng.uniform(0, 1.5))
    return _cloud(*_scan(boxes, poles, np.eye(4), n, _gen(seed, 1))), _cloud(*_scan(boxes, poles, S, n, _gen(seed, 2))), S


def _near(T, rng, deg, dist):
    """A pose `deg` degrees and `dist` metres off T, as a motion prior is."""
    return (T @ scenes.make_T(scenes.rot_axis_angle(_unit(rng), math.radians(deg)), _unit(rng) * dist)).astype(np.float32)


# ----------------------------------------------------------------- prepare
def _params(case):
    p = CvoParams(params_path("irls" if case["kind"] == "window" else PARAMS[case.get("scene", "color")]))
    p.ell_init = case.get("ell", p.ell_init)
    p.MAX_ITER = case.get("iters", p.MAX_ITER)
    p.nearest_neighbors_max = case.get("cap", p.nearest_neighbors_max)
    p.multiframe_max_iters = case.get("outer", p.multiframe_max_iters)
    return p


def _inputs(case, seed):
    """Host inputs of a case, from the seed alone."""
    kind, rng = case["kind"], np.random.default_rng([seed, 5])
    if kind == "rgbd":
        r, c, n = case["rows"], case["cols"], case["n"]
        y, x = np.mgrid[0:r, 0:c]
        ph = rng.uniform(0, 2 * np.pi, 6)
        img = np.stack([127.5 + 100 * np.sin(x / (9.0 + k) + ph[k]) * np.cos(y / (7.0 + k) + ph[3 + k]) for k in range(3)], 2)
        img = (img + rng.uniform(-20, 20, img.shape)).clip(0, 255).astype(np.uint8)
        depth = (1000 * (6 + 4 * np.sin(x / 90.0 + ph[0]) * np.cos(y / 70.0) + rng.uniform(0, 0.05, (r, c)))).astype(np.float32)
        pix = rng.choice(r * c, size=min(n, r * c), replace=False)
        depth.reshape(-1)[pix[: len(pix) // 20]] = 0.0   # no return at some of the selected pixels
        pix = np.sort(pix)
        return {"img": img, "depth": depth, "uv": np.stack([pix % c, pix // c], 1).astype(np.int32),
                "K": np.array([0.58 * c, 0.58 * c, c / 2, r / 2], np.float32)}
    if kind == "train":
        views = []
        for k in range(8):
            w = scenes._TexturedWorld(np.random.default_rng([seed, k]))
            a, b = _view(w, np.eye(4), 2048, _gen(seed, 2 * k)), _view(w, np.eye(4), 2048, _gen(seed, 2 * k + 1))
            m = a[0].mean(0)
            views.append([torch.cat([q - m, f], 1).to(torch.float32).cpu().numpy() for q, f in (a, b)])
        T = np.stack([scenes.random_motion(rng) for _ in range(case["pairs"])]).astype(np.float32)
        return {"src": np.stack([v[0] for v in views]), "tgt": np.stack([v[1] for v in views]),
                "scene": rng.integers(0, 8, case["pairs"]).astype(np.int32), "T": T, "seed": int(rng.integers(1 << 31))}
    if kind == "window":
        w, F = scenes._TexturedWorld(rng, n_patches=64), case["frames"]
        poses, yaw = [np.eye(4)], 0.0
        for _ in range(1, F):
            yaw += math.radians(rng.uniform(-2, 2))
            poses.append(scenes.make_T(scenes.rot_axis_angle([0, 1, 0], yaw), poses[-1][:3, 3] + 0.8 * poses[-1][:3, 2]))
        clouds = [_cloud(*_view(w, T, int(rng.integers(case["lo"], case["hi"] + 1)), _gen(seed, k))) for k, T in enumerate(poses)]
        start = [poses[0]] + [_near(T, rng, 0.15, 0.03) for T in poses[1:]]
        return {"clouds": clouds, "poses": np.stack([T[:3].reshape(12) for T in start]).astype(np.float64),
                "hold": np.array([1] + [0] * (F - 1), np.uint8),
                "edges": np.array([[i, j] for i in range(F) for j in range(i + 1, F)], np.int32)}
    if kind == "align_batch":
        sizes = [max(1000, int(case["n"] * rng.uniform(0.4, 1.0))) for _ in range(case["pairs"])]
        pairs = [_pair("color", n, seed * 31 + k) for k, n in enumerate(sizes)]
        # hypotheses of the proposal network end up within some degrees
        return {"pairs": pairs, "T": [np.linalg.inv(_near(G, rng, rng.uniform(0.5, 3), 0.1)) for _, _, G in pairs]}
    s, t, G = _pair(case["scene"], case["n"], seed)
    if kind == "cos":
        T = [scenes.make_T(R, _unit(rng) * 0.2).astype(np.float32) for R in CvoGPU.rotation_grid(0)[:case["poses"]]]
    elif kind.startswith("align"):
        T = np.linalg.inv(_near(G, rng, 0.5, 0.1))
    else:
        T = np.linalg.inv(_near(G, rng, 0.3, 0.03))
    return {"s": s, "t": t, "T": T}


def prepare(case, seed):
    x = _inputs(case, seed)
    x["kind"] = kind = case["kind"]
    cvo = x["cvo"] = CvoGPU(params=_params(case))
    if kind in ("cos", "align", "aniso"):
        x["ds"], x["dt"] = cvo.upload(x["s"]), cvo.upload(x["t"])
    elif kind == "align_batch":
        x["ds"], x["dt"] = [cvo.upload(s) for s, _, _ in x["pairs"]], [cvo.upload(t) for _, t, _ in x["pairs"]]
    elif kind == "window":
        x["dev"] = [cvo.upload(c) for c in x["clouds"]]
    elif kind == "train":
        x["net"] = ProposalNet(cvo, points_per_cloud=case["points"], seed=7)
        x["pool"] = ScenePool(x["src"], x["tgt"])
    if kind in ("assoc", "aniso"):   # the back end's correspondence buffers: a fixed number of each point
        x["col"], x["val"] = np.zeros(len(x["s"]) * case["cap"], np.int32), np.zeros(len(x["s"]) * case["cap"], np.float32)
    x["ell"] = case.get("ell")
    return x


def _kernel3():
    return np.diag([0.5, 0.5, 0.6]).astype(np.float32)


def run(x):
    cvo, kind = x["cvo"], x["kind"]
    if kind == "ip":
        return {"ip": cvo.inner_product_gpu(x["s"], x["t"], x["T"], x["ell"])}
    if kind == "cos":
        return {"ip": cvo.inner_product_batch(x["ds"], x["dt"], x["T"], x["ell"])}
    if kind in ("align", "align_host"):
        on = ("ds", "dt") if kind == "align" else ("s", "t")
        ret, T, _, _, _ = cvo.align(x[on[0]], x[on[1]], x["T"])
        return {"T": T, "ret": ret}
    if kind == "align_batch":
        T, rets, _, _ = cvo.align_batch(x["ds"], x["dt"], x["T"])
        return {"T": T, "ret": rets}
    if kind in ("assoc", "aniso"):
        if kind == "assoc":
            a = cvo.compute_association_gpu(x["s"], x["t"], x["T"], x["ell"])
        else:
            a = cvo.compute_association_gpu(x["ds"], x["dt"], x["T"], _kernel3())
        for name in ("col", "val"):
            x[name][:a.nnz] = getattr(a, name)
            x[name][a.nnz:] = 0
        return {"row_ptr": a.row_ptr, "col": x["col"], "val": x["val"]}
    if kind == "rgbd":
        c = cvo.cloud_from_rgbd(x["img"], x["depth"], x["K"], 1000.0, x["uv"]).download()
        return {"xyz": c.xyz, "features": c.features}
    if kind == "window":
        # poses to float, as the next association and the map take them
        return {"poses": cvo.align_multi(x["dev"], x["poses"], x["hold"], x["edges"])[0].astype(np.float32)}
    net = x["net"]
    loss = net.train_step(x["pool"], x["scene"], x["T"], 1e-3, x["seed"])
    return {"loss": loss, "gradients": net.gradients(), "weights": net.weights()}


# -------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "rgbd":
        return {"bytes": case["rows"] * case["cols"] * 7 + case["n"] * (8 + 2 * 32 + 32), "flops": 40.0 * case["n"]}
    if kind == "train":
        rows = 2 * case["pairs"] * case["points"]
        macs = rows * (8 * 64 + 64 * 128) + case["pairs"] * (256 * 256 + 256 * 72)
        return {"bytes": 4.0 * (rows * 8 + 6 * 93704), "flops": 6.0 * macs}
    rec = RECORD[case.get("scene", "color")]
    if kind == "window":
        n = 0.5 * (case["lo"] + case["hi"])
        E = case["frames"] * (case["frames"] - 1) / 2
        # each outer iteration: every edge's clouds once, its kept pairs evaluated and entered in the normal equations
        return {"bytes": case["outer"] * E * 2 * n * rec, "flops": case["outer"] * E * n * 40 * (40 + 220.0)}
    n, kept = case["n"], {"room": 60, "color": 120, "lidar": 60}[case["scene"]]
    passes = case.get("iters", 1) * case.get("pairs", 1) * case.get("poses", 1)
    per = 40.0 + (110.0 if kind.startswith("align") else 0.0)   # kernel value; gradient and step-size terms
    out = 8.0 * n * kept if kind in ("assoc", "aniso") else 0.0
    return {"bytes": passes * 2.0 * n * rec + out, "flops": passes * per * n * kept}


# ------------------------------------------------------------------- exact
def _f(v):
    """A parameter in 64 bits, from its 32-bit value."""
    return float(np.float32(v))


def _dense(c):
    if c is None:
        return None
    return _t(c.astype(np.float64))


class _Kernel:
    """The kernel matrix between x (n, 3) and y (m, 3): pairs above the threshold, the first cap of each row."""

    def __init__(self, p, s, t):
        self.p, self.fs, self.ft, self.ls, self.lt = p, _dense(s.features), _dense(t.features), _dense(s.labels), _dense(t.labels)
        self.use_f, self.use_l = bool(p.is_using_intensity), bool(p.is_using_semantics)
        c, s_ = _f(p.c_ell), _f(p.s_ell)
        side = [[f / (math.sqrt(2) * w) for f, w, on in ((f, c, self.use_f), (l, s_, self.use_l)) if on]
                for f, l in ((self.fs, self.ls), (self.ft, self.lt))]
        self.a, self.b = (torch.cat(q, 1) if q else None for q in side)
        sp = _f(p.sp_thres)
        self.geo2, self.c2, self.s2 = _f(p.sigma) ** 2, _f(p.c_sigma) ** 2, _f(p.s_sigma) ** 2
        self.scale = self.geo2 * (self.c2 if self.use_f else 1.0) * (self.s2 if self.use_l else 1.0)
        self.tau, self.sp = math.log(self.scale / sp), sp
        self.log_geo = math.log(sp / self.geo2)
        self.dc = -2 * c * c * math.log(sp / self.c2)
        self.ds = -2 * s_ * s_ * math.log(sp / self.s2)

    def pairs(self, x, y, ell, cap, step=1 << 28):
        """(i, j, value) of the kept pairs, rows ascending, columns ascending."""
        l = (x.norm(dim=1) / 500.0 + 1.0) * ell
        g = 1.0 / (2 * l * l)
        one = torch.ones_like(g)[:, None]
        A = [-2 * g[:, None] * x, g[:, None], (g * (x * x).sum(1))[:, None]]
        B = [y, (y * y).sum(1, keepdim=True), torch.ones_like(y[:, :1])]
        if self.a is not None:
            A = A[:2] + [A[2] + (self.a ** 2).sum(1, keepdim=True), -2 * self.a, one]
            B += [self.b, (self.b ** 2).sum(1, keepdim=True)]
        A, B = torch.cat(A, 1), torch.cat(B, 1).T.contiguous()
        out, rows = [], max(1, step // y.shape[0])
        for r0 in range(0, x.shape[0], rows):
            i, j = ((A[r0:r0 + rows] @ B) < self.tau + 1e-6).nonzero(as_tuple=True)
            i = i + r0
            d2 = ((x[i] - y[j]) ** 2).sum(1)
            keep = d2 < -2 * l[i] ** 2 * self.log_geo
            v = self.scale * torch.exp(-d2 * g[i])
            if self.use_f:
                e = ((self.fs[i] - self.ft[j]) ** 2).sum(1)
                keep &= e < self.dc
                v = v * torch.exp(-e / (2 * _f(self.p.c_ell) ** 2))
            if self.use_l:
                e = ((self.ls[i] - self.lt[j]) ** 2).sum(1)
                keep &= e < self.ds
                v = v * torch.exp(-e / (2 * _f(self.p.s_ell) ** 2))
            out.append(_first(i, j, v, keep & (v > self.sp), cap, x.shape[0]))
        return [torch.cat(c) for c in zip(*out)]


def _first(i, j, v, keep, cap, n):
    """The kept pairs, at most the first cap of each row (pairs come in row, column order)."""
    i, j, v = i[keep], j[keep], v[keep]
    start = torch.searchsorted(i, torch.arange(n, device=i.device))
    few = torch.arange(len(i), device=i.device) - start[i] < cap
    return i[few], j[few], v[few]


def _skew(w):
    return np.array([[0, -w[2], w[1]], [w[2], 0, -w[0]], [-w[1], w[0], 0]])


def _exp(w, v, dt=1.0):
    """exp of dt (w, v) as 4 x 4."""
    th, A = np.linalg.norm(w), _skew(w)
    if th < 1e-12:
        return scenes.make_T(np.eye(3), dt * np.asarray(v))
    R = np.eye(3) + math.sin(dt * th) / th * A + (1 - math.cos(dt * th)) / th ** 2 * A @ A
    J = dt * np.eye(3) + (1 - math.cos(dt * th)) / th ** 2 * A + (dt * th - math.sin(dt * th)) / th ** 3 * A @ A
    return scenes.make_T(R, J @ v)


def _log_norm(T):
    w = np.array([T[2, 1] - T[1, 2], T[0, 2] - T[2, 0], T[1, 0] - T[0, 1]]) / 2
    s = np.linalg.norm(w)
    th = math.atan2(s, (np.trace(T[:3, :3]) - 1) / 2)
    if th < 1e-9:
        return float(np.linalg.norm(T[:3, 3]))
    w = w * th / s
    A = _skew(w)
    u = T[:3, 3] - 0.5 * A @ T[:3, 3] + (1 / th ** 2 - (1 + math.cos(th)) / (2 * th * math.sin(th))) * A @ A @ T[:3, 3]
    return math.sqrt(u @ u + th * th)


class _Indicator:
    """Two adjacent windows over the sparsity of the kernel matrix: stable when their sums agree."""

    def __init__(self, length, tol):
        self.n, self.tol, self.a, self.b = length, tol, [], []

    def update(self, v):
        if len(self.a) < self.n:
            self.a.append(v)
        if len(self.a) >= self.n and len(self.b) < self.n:
            self.b.append(v)
        if len(self.a) < self.n or len(self.b) < self.n:
            return False
        if 1 - self.tol < sum(self.b) / sum(self.a) < 1 + self.tol:
            self.a, self.b = [], []
            return True
        self.a = self.a[1:] + [self.b[0]]
        self.b = self.b[1:] + [v]
        return False


def _step(x, z, i, a, ell, w, v, lo, hi):
    """Step length along the twist (w, v): smallest positive root of the objective's quartic model's derivative."""
    w, v = _t(w), _t(v)
    c = 1.0 / (2 * ell * ell)
    cr = lambda q: torch.linalg.cross(w.expand_as(q), q)  # noqa: E731
    u = cr(z) + v
    p = cr(u)
    q = cr(p)
    r = cr(q)
    d = x[i] - z
    dot = lambda s, t: (s * t).sum(1)  # noqa: E731
    be = -2 * c * dot(u, d)
    ga = -c * (dot(u, u) + 2 * dot(p, d))
    de = 2 * c * (-dot(u, p) - dot(q, d))
    ep = -c * (dot(p, p) + 2 * dot(u, q) + 2 * dot(r, d))
    co = [be, ga + be ** 2 / 2, de + be * ga + be ** 3 / 6, ep + be * de + be ** 2 * ga / 2 + ga ** 2 / 2 + be ** 4 / 24]
    b = [float((a * t).sum()) for t in co]
    roots = [z.real for z in np.roots([4 * b[3], 3 * b[2], 2 * b[1], b[0]]) if abs(z.imag) < 1e-5 and z.real > 0] if b[3] else []
    return min(max(min(roots, default=math.inf), lo), hi)


def _exact_align(p, s, t, T0):
    k, x, y0 = _Kernel(p, s, t), _dense(s.xyz), _dense(t.xyz)
    T = np.asarray(np.float32(T0), np.float64)
    ell, cap, ind = _f(p.ell_init), p.nearest_neighbors_max, _Indicator(p.indicator_window_size, _f(p.indicator_stable_threshold))
    for it in range(p.MAX_ITER):
        y = (y0 - _t(T[:3, 3])) @ _t(T[:3, :3])
        i, j, a = k.pairs(x, y, ell, cap)
        z = y[j]
        w = (a[:, None] * torch.linalg.cross(x[i], z)).sum(0).cpu().numpy() / _f(p.c)
        v = (a[:, None] * (z - x[i])).sum(0).cpu().numpy() / _f(p.d)
        g = math.sqrt(w @ w + v @ v)
        if g == 0:
            break
        w, v = w / g, v / g
        dT = _exp(w, v, _step(x, z, i, a, ell, w, v, _f(p.min_step), _f(p.max_step)))
        T = T @ dT
        decay = ind.update(len(a) / math.sqrt(len(x) * len(y0)))
        if _log_norm(dT) < _f(p.eps_2):
            break
        if it > p.ell_decay_start and decay:
            ell = max(_f(p.ell_min), ell * _f(p.ell_decay_rate))
        cap = min(p.nearest_neighbors_max, int(int(torch.bincount(i).max()) * 1.2))
    return np.linalg.inv(T)


def _exact_aniso(p, s, t, T):
    k, x = _Kernel(p, s, t), _dense(s.xyz)
    T = _t(np.float32(T).astype(np.float64))
    y = (_dense(t.xyz) - T[:3, 3]) @ T[:3, :3]
    z = x / x.norm(dim=1, keepdim=True)
    e = torch.stack([torch.ones_like(z[:, 0]), torch.ones_like(z[:, 0]), -(z[:, 0] + z[:, 1]) / z[:, 2]], 1)
    U = torch.stack([e, torch.linalg.cross(z, e), z], 2)
    M = U @ torch.linalg.inv(_t(_kernel3().astype(np.float64))) @ U.transpose(1, 2)
    out, rows = [], 1000
    for r0 in range(0, len(x), rows):
        dc = torch.cdist(k.a[r0:r0 + rows], k.b)
        i, j = (dc * dc < k.tau + 1e-6).nonzero(as_tuple=True)
        i = i + r0
        d = x[i] - y[j]
        ec = ((k.fs[i] - k.ft[j]) ** 2).sum(1)
        v = k.scale * torch.exp(-0.5 * ((d[:, None] @ M[i])[:, 0] * d).sum(1)) * torch.exp(-ec / (2 * _f(p.c_ell) ** 2))
        out.append(_first(i, j, v, (ec < k.dc) & (v > k.sp), p.nearest_neighbors_max, len(x)))
    return [torch.cat(c) for c in zip(*out)]


def _exact_window(p, x):
    """The window solve: kernel matrices of every edge, then Levenberg-Marquardt on a |T1 p1 - T2 p2|^2."""
    C = [_dense(c.xyz) for c in x["clouds"]]
    T = [np.vstack([q.reshape(3, 4), [0, 0, 0, 1]]) for q in x["poses"]]
    E, F = x["edges"], len(C)
    kern = [_Kernel(p, x["clouds"][i], x["clouds"][j]) for i, j in E]
    free = [f for f in range(F) if not x["hold"][f]]
    ell, cap = [_f(p.multiframe_ell_init)] * len(E), [p.multiframe_num_neighbors] * len(E)
    most, nnz, held = [0] * len(E), [0] * len(E), [0] * len(E)
    for _ in range(p.multiframe_max_iters):
        old, before = [q.copy() for q in T], list(nnz)
        W = [c @ _t(np.float32(q[:3, :3]).astype(np.float64)).T + _t(np.float32(q[:3, 3]).astype(np.float64)) for c, q in zip(C, T)]
        kept = []
        for e, (f1, f2) in enumerate(E):
            if most[e] > 0:
                cap[e] = min(p.multiframe_num_neighbors, int(most[e] * 1.1))
            i, j, a = kern[e].pairs(W[f1], W[f2], ell[e], cap[e])
            nnz[e], most[e] = len(a), int(torch.bincount(i).max()) if len(a) else 0
            if len(a) and len(a) >= p.multiframe_min_nonzeros:
                kept.append((f1, f2, C[f1][i], C[f2][j], a))
        if not any(v > p.multiframe_min_nonzeros for v in nnz):
            break

        def cost(T, want):
            H, g, c = np.zeros((6 * F, 6 * F)), np.zeros(6 * F), 0.0
            for f1, f2, p1, p2, a in kept:
                R1, R2 = _t(T[f1][:3, :3]), _t(T[f2][:3, :3])
                d = p1 @ R1.T + _t(T[f1][:3, 3]) - p2 @ R2.T - _t(T[f2][:3, 3])
                r = a * (d * d).sum(1)
                c += 0.5 * float((r * r).sum())
                if want:
                    u1, u2 = d @ R1, d @ R2
                    J = torch.cat([u1, torch.linalg.cross(p1, u1), -u2, -torch.linalg.cross(p2, u2)], 1)
                    at = np.r_[6 * f1:6 * f1 + 6, 6 * f2:6 * f2 + 6]
                    H[np.ix_(at, at)] += (J.T @ J).cpu().numpy()
                    g[at] += (J.T @ r).cpu().numpy()
            return H, g, c

        at = np.concatenate([np.arange(6 * f, 6 * f + 6) for f in free])
        radius, nu = 1e4, 2.0
        H, g, c = cost(T, True)
        for _ in range(p.multiframe_iterations_per_solve):
            Hf, gf = H[np.ix_(at, at)], g[at]
            if np.abs(gf).max() <= 1e-5:
                break
            b = np.linalg.solve(Hf + np.diag(np.clip(np.diag(Hf), 1e-6, 1e32)) / radius, -gf)
            if np.linalg.norm(b) <= 1e-5 * (math.sqrt(sum((q[:3] ** 2).sum() for q in T)) + 1e-5):
                break
            new = [q.copy() for q in T]
            for k, f in enumerate(free):
                new[f] = T[f] @ _exp(b[6 * k + 3:6 * k + 6], b[6 * k:6 * k + 3])
            model = -(gf @ b + 0.5 * b @ Hf @ b)
            cn = cost(new, False)[2]
            rho = (c - cn) / model if model > 0 else -1.0
            if rho > 1e-3:
                T, stop = new, abs(c - cn) <= 1e-5 * c
                radius, nu = radius / max(1 / 3, 1 - (2 * rho - 1) ** 3), 2.0
                if stop:
                    break
                H, g, c = cost(T, True)
            else:
                radius, nu = radius / nu, 2 * nu
        lo, hi = _f(p.multiframe_ell_min), 1.2 * _f(p.multiframe_ell_init)
        for e in range(len(E)):
            held[e] += 1
            if before[e] > 0 and nnz[e] <= before[e] and held[e] // p.multiframe_iter_per_ell > 0:
                ell[e], held[e] = ell[e] * _f(p.multiframe_ell_decay_rate), 0
            ell[e] = min(max(ell[e], lo), hi)
        change = sum(_log_norm(np.linalg.inv(a) @ b) for a, b in zip(old, T))
        if all(abs(l - lo) < 1e-4 for l in ell) and change < 1e-5:
            break
    return np.stack([q[:3].reshape(12) for q in T])


def _mix(v):
    for s, m in ((16, 0x7FEB352D), (15, 0x846CA68B), (16, 1)):
        v = v ^ (v >> s)
        v = (v * m) & 0xFFFFFFFF
    return v


def _exact_train(case, x, w0):
    shapes = [(16, 64), (64,), (64, 128), (128,), (256, 256), (256,), (256, 72), (72,)]
    w = _t(w0.astype(np.float64)).requires_grad_()
    W1, b1, W2, b2, W3, b3, W4, b4 = [q.reshape(s) for q, s in zip(w.split([math.prod(s) for s in shapes]), shapes)]
    B, P, n = case["pairs"], case["points"], x["src"].shape[1]
    X, cent = [], []
    for b in range(B):
        for side, pool in ((0, x["src"]), (1, x["tgt"])):
            pts = pool[x["scene"][b]].astype(np.float64)
            T = np.eye(4)[:3] if side == 0 else x["T"][b].astype(np.float64)
            m, slot = pts[:, :3].mean(0), 2 * b + side
            h = _mix(np.uint64(_mix((x["seed"] + 0x9E3779B9 * (slot + 1)) & 0xFFFFFFFF)) ^ np.arange(P, dtype=np.uint64))
            q = pts[((h * np.uint64(n)) >> np.uint64(32)).astype(np.int64)]
            X.append(np.concatenate([0.1 * (q[:, :3] - m) @ T[:, :3].T, q[:, 3:], np.zeros((P, 8))], 1))
            cent.append(T[:, :3] @ m + T[:, 3])
    X, cent = _t(np.stack(X)), np.stack(cent).reshape(B, 2, 3)
    H = torch.relu(torch.relu(X @ W1 + b1) @ W2 + b2)
    G = H.amax(1).reshape(B, 256)
    O = (torch.relu(G @ W3 + b3) @ W4 + b4).reshape(B, 8, 9)
    R, t = x["T"][:, :, :3].astype(np.float64), x["T"][:, :, 3].astype(np.float64)
    y = np.concatenate([R[:, :, 0], R[:, :, 1], 0.1 * (t - cent[:, 1] + (R @ cent[:, 0, :, None])[..., 0])], 1)
    L = ((O - _t(y)[:, None]) ** 2).sum(-1)
    wt = torch.full_like(L, 0.05 / 7).scatter(1, L.argmin(1, keepdim=True), 0.95)
    loss = (wt * L).sum(1).mean()
    g = torch.autograd.grad(loss, w)[0]
    return {"loss": float(loss), "gradients": g, "weights": w.detach() - 1e-3 * g / (g.abs() + 1e-8)}


def _padded(case, x, v):
    return {"row_ptr": None, "col": None, "val": torch.cat([v, v.new_zeros(len(x["s"]) * case["cap"] - len(v))])}


def exact(case, seed):
    x, kind, p = _inputs(case, seed), case["kind"], _params(case)
    if kind == "rgbd":
        I = x["img"].astype(np.float64)
        grey = np.floor((1868 * I[..., 0] + 9617 * I[..., 1] + 4899 * I[..., 2] + 8192) / 16384)
        grad = np.zeros(grey.shape + (2,))
        grad[1:-1, 1:-1, 0] = 0.5 * (grey[1:-1, 2:] - grey[1:-1, :-2])
        grad[1:-1, 1:-1, 1] = 0.5 * (grey[2:, 1:-1] - grey[:-2, 1:-1])
        u, v = x["uv"].T.astype(np.int64)
        fx, fy, cx, cy = x["K"].astype(np.float64)
        z = x["depth"][v, u].astype(np.float64) / 1000.0
        q = np.stack([(u - cx) * z / fx, (v - cy) * z / fy, z], 1)
        ok = (z != 0) & (np.linalg.norm(q, axis=1) <= 55)
        gf, at = grad.reshape(-1), v * x["img"].shape[1] + u
        f = np.concatenate([I[v, u] / 255.0, np.stack([gf[at], gf[at + 1]], 1) / 500.0 + 0.5], 1)
        return {"xyz": q[ok], "features": f[ok]}
    if kind == "train":
        return _exact_train(case, x, ProposalNet(CvoGPU(params=p), points_per_cloud=case["points"], seed=7).weights())
    if kind == "window":
        return {"poses": _exact_window(p, x)}
    if kind == "align_batch":
        if case["pairs"] * case["iters"] * case["n"] ** 2 > 2e11:   # minutes of 64-bit arithmetic
            return None
        return {"T": [_exact_align(p, s, t, T) for (s, t, _), T in zip(x["pairs"], x["T"])], "ret": None}
    if kind.startswith("align"):
        return {"T": _exact_align(p, x["s"], x["t"], x["T"]), "ret": None}
    if kind == "aniso":
        return _padded(case, x, _exact_aniso(p, x["s"], x["t"], x["T"])[2])
    k, a, b, ips = _Kernel(p, x["s"], x["t"]), _dense(x["s"].xyz), _dense(x["t"].xyz), []
    for T in x["T"] if kind == "cos" else [x["T"]]:
        T = _t(np.float32(T).astype(np.float64))
        v = k.pairs(a, (b - T[:3, 3]) @ T[:3, :3], _f(case["ell"]), p.nearest_neighbors_max)[2]
        ips.append(float(v.sum()))
    if kind == "assoc":
        return _padded(case, x, v)
    return {"ip": np.array(ips) if kind == "cos" else ips[0]}
