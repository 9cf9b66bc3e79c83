"""The sphere-tracing work a program has this library do, as cases that can be timed.

Every case goes through the public entry points (``runtime.Context``): a forward march
of one view or a batch of views into a G-buffer, the same recorded as a graph, the FP64
march of a close-up, lite shading of a frame, the empty-space accelerator, a
differentiation step (forward, loss, adjoint), and the DE at points.  The formula is the
package's own ``mandelbulb_bailout``, which every build has.  Sizes are those of the
package's workloads (``workloads.py``: 256 x 256, 1920 x 1080, 64 views with sides of 64
to 1024 pixels, 512 x 512 differentiation problems) and ordinary frame sizes.

The inputs of a case (cameras, powers, lights, loss targets, points) come from the seed.
``exact`` restates the march, the normals, the orbit trap, the shadow ray, the lite
shading and the adjoint in FP64 torch, without the package's kernels.
"""

import math
import random

import numpy as np
import torch

from numericdream_b200 import abi, runtime

FORMULA = "mandelbulb_bailout"
LIGHT = (0.4, 0.8, -0.45)
STOPS = [((0.05, 0.05, 0.22), 0.0, 0.2, 1.3), ((0.85, 0.35, 0.08), 0.5, 0.5, 1.5), ((1.0, 0.95, 0.82), 1.0, 0.8, 1.7)]
LIGHTS = [(abi.ND_LIGHT_GLOBAL, (0.4, 0.8, -0.45), (1.0, 0.95, 0.9), 1.2),
          (abi.ND_LIGHT_POINT, (2.0, 2.5, -3.0), (0.6, 0.7, 1.0), 6.0)]


def listed():
    return [
        # a scene list's thumbnail: the smallest call, where latency and launches count
        {"name": "thumb_96x54", "kind": "view", "w": 96, "h": 54, "spp": 1, "iters": 12, "steps": 256, "style": "plain"},
        # the interactive preview while a slider moves (the package's 256 x 256 view)
        {"name": "preview_256", "kind": "view", "w": 256, "h": 256, "spp": 1, "iters": 12, "steps": 256, "style": "plain"},
        # a final-quality export: verified steps, hq footprint, tetrahedral normals, odd frame
        {"name": "export_hq_843x611", "kind": "view", "w": 843, "h": 611, "spp": 1, "iters": 10, "steps": 384,
         "style": "hq"},
        # an antialiased full-HD frame with soft shadows (the package's 1080p options)
        {"name": "shadow_1080p_2spp", "kind": "view", "w": 1920, "h": 1080, "spp": 2, "iters": 12, "steps": 512,
         "style": "shadow"},
        # the renderer's batch: 64 views, uneven sides, the reference's G-buffer formats
        {"name": "batch_64", "kind": "batch", "views": 64, "min": 64, "max": 1024, "iters": 6, "steps": 384},
        # a contact sheet of a few odd views
        {"name": "batch_7", "kind": "batch", "views": 7, "min": 61, "max": 317, "iters": 12, "steps": 256},
        # an animation loop that replays a captured graph of small views
        {"name": "graph_8", "kind": "graph", "views": 8, "min": 96, "max": 160, "iters": 8, "steps": 256},
        # a close-up that an FP32 DE cannot resolve: FP64 DE and ray directions, 20 bisections
        {"name": "closeup_fp64_512", "kind": "closeup", "w": 512, "h": 512, "iters": 14, "fov": 0.1, "standoff": 1e-3},
        # a shaded frame: forward and lite shading (colour strip, AO, two lights)
        {"name": "lite_1280x720", "kind": "lite", "w": 1280, "h": 720, "iters": 10, "steps": 256},
        # a frame with the empty-space accelerator at the reference's default grid
        {"name": "accel_960x540", "kind": "accel", "w": 960, "h": 540, "iters": 10, "steps": 256, "res": 64},
        # inverse rendering: forward, loss and FP32 adjoint of several problems at once
        {"name": "diff_fp32_4x512", "kind": "diff", "problems": 4, "side": 512, "iters": 12, "precision": 32},
        # the same in FP64 with the per-ray Jacobian (Gauss-Newton steps)
        {"name": "diff_fp64_2x256", "kind": "diff", "problems": 2, "side": 256, "iters": 12, "precision": 64},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["view", "view", "view", "batch", "batch", "graph", "closeup", "lite", "accel", "diff", "diff"])
    c = {"kind": kind, "iters": rng.randint(6, 14)}
    if kind == "view":
        c["style"] = rng.choice(["plain", "hq", "shadow"])
        c["w"], c["h"] = log(64, 1920), log(48, 1080)
        c["spp"] = rng.choice([1, 1, 2])
        c["steps"] = rng.choice([128, 256, 384, 512])
    elif kind in ("batch", "graph"):
        c["views"] = log(2, 64) if kind == "batch" else log(2, 12)
        c["min"] = rng.randint(33, 90)
        c["max"] = c["min"] + log(20, 500 if kind == "batch" else 200)
        c["iters"] = rng.randint(5, 12)
        c["steps"] = rng.choice([192, 256, 384])
    elif kind == "closeup":
        c["w"], c["h"] = log(96, 512), log(96, 512)
        c["fov"] = round(math.exp(rng.uniform(math.log(0.05), math.log(5.0))), 4)
        c["standoff"] = round(math.exp(rng.uniform(math.log(1e-3), math.log(1e-1))), 6)
    elif kind in ("lite", "accel"):
        c["w"], c["h"] = log(160, 1280), log(120, 720)
        c["steps"] = rng.choice([128, 256, 384])
        if kind == "accel":
            c["res"] = rng.choice([16, 32, 48, 64])
    else:
        c["problems"], c["side"] = rng.randint(1, 4), log(64, 360)
        c["precision"] = rng.choice([32, 32, 64])
    return c


# ---------------------------------------------------------------- inputs
_ctx = []


def _context():
    if not _ctx:
        _ctx.append(runtime.Context(0))
    return _ctx[0]


def _orbit_position(rng, dist):
    yaw, pitch = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(-0.6, 0.6)
    return (dist * math.cos(pitch) * math.sin(yaw), dist * math.sin(pitch), -dist * math.cos(pitch) * math.cos(yaw))


def _power(rng):
    # the sliders step through whole powers more often than not
    return float(rng.choice([4, 5, 6, 7, 8, 8, 8, 9, 10])) if rng.random() < 0.6 else rng.uniform(4.0, 10.0)


def _views(case, seed):
    """The case's views (and its orbit cameras, for the differentiation cases)."""
    rng = random.Random(seed * 7919 + 11)
    kind = case["kind"]
    fid = runtime.find_formula(FORMULA)
    central = {"normal_mode": abi.ND_NORMAL_CENTRAL, "normal_h_coef": 1e-4}
    sphere = {"shape": abi.ND_TRAP_SPHERE, "radius": 1.0}
    if kind == "view" and case["style"] == "plain":
        return [abi.make_view(fid, case["w"], case["h"], _orbit_position(rng, 2.5 + 0.02 * rng.random()), fov_y_deg=60.0,
                              params=[8.0, case["iters"], 2.0], spp=case["spp"], seed=seed, max_steps=case["steps"],
                              eps_coef=1e-4, eps_floor=0.0, trap=sphere, **central)], None
    if kind == "view" and case["style"] == "hq":
        return [abi.make_view(fid, case["w"], case["h"], _orbit_position(rng, 2.4 + 0.02 * rng.random()), fov_y_deg=55.0,
                              params=[8.0, case["iters"], 2.0], spp=case["spp"], seed=seed, max_steps=case["steps"],
                              refine_budget=20, march_verify=1, high_quality=1)], None
    if kind == "view":
        return [abi.make_view(fid, case["w"], case["h"], _orbit_position(rng, 2.2 + 0.02 * rng.random()), fov_y_deg=70.0,
                              params=[8.0, case["iters"], 2.0], spp=case["spp"], seed=seed, max_steps=case["steps"],
                              eps_coef=5e-5, eps_floor=0.0, normal_mode=abi.ND_NORMAL_CENTRAL, shadow=1,
                              light_dir=list(LIGHT), shadow_k=16.0,
                              trap={"shape": abi.ND_TRAP_BOX, "box": [1.0, 1.0, 1.0]})], None
    if kind in ("batch", "graph"):
        shape = random.Random(case["views"] * 1000 + case["max"])  # the sizes are the case's, not the seed's
        views = []
        for i in range(case["views"]):
            w, h = (int(round(math.exp(shape.uniform(math.log(case["min"]), math.log(case["max"]))))) for _ in range(2))
            views.append(abi.make_view(fid, w, h, _orbit_position(rng, rng.uniform(1.8, 4.0)), fov_y_deg=60.0,
                                       params=[_power(rng), case["iters"], 2.0], max_steps=case["steps"],
                                       seed=seed * 1000 + i, trap=sphere, **central))
        return views, None
    if kind == "closeup":
        power = float(rng.choice([6, 8, 8, 9]))
        org, d, t = _surface_ray(rng, power, case["iters"])
        cam = [org[i] + d[i] * (t - case["standoff"]) for i in range(3)]
        return [abi.make_view(fid, case["w"], case["h"], cam, target=[cam[i] + d[i] for i in range(3)],
                              fov_y_deg=case["fov"], params=[power, case["iters"], 2.0], max_steps=512, max_dist=1.0,
                              eps_coef=1e-6, eps_floor=0.0, refine_budget=20, normal_mode=abi.ND_NORMAL_CENTRAL,
                              normal_h_coef=1e-6, flags=abi.ND_VIEW_DIR64)], None
    if kind == "lite":
        return [abi.make_view(fid, case["w"], case["h"], _orbit_position(rng, 2.6 + 0.02 * rng.random()), fov_y_deg=60.0,
                              params=[8.0, case["iters"], 2.0], max_steps=case["steps"],
                              trap={"shape": abi.ND_TRAP_SPHERE, "radius": 1.0, "span": 0.8, "repeat": 2})], None
    if kind == "accel":
        return [abi.make_view(fid, case["w"], case["h"], _orbit_position(rng, 2.6 + 0.02 * rng.random()), fov_y_deg=60.0,
                              params=[8.0, case["iters"], 2.0], max_steps=case["steps"], accel_res=case["res"],
                              accel_levels=6, trap=sphere, **central)], None
    views, cams = [], []
    for _ in range(case["problems"]):
        cam = abi.orbit_camera(yaw=rng.uniform(-0.6, 0.6), pitch=rng.uniform(-0.3, 0.3), dist=2.5, fov_y_deg=60.0)
        v = abi.make_view(fid, case["side"], case["side"], (0.0, 0.0, -2.5), fov_y_deg=60.0,
                          params=[rng.uniform(6.0, 10.0), case["iters"], 2.0], max_steps=256, eps_coef=1e-4,
                          eps_floor=0.0, refine_budget=40, light_dir=list(LIGHT), flags=abi.ND_VIEW_EXACT_HIT, **central)
        runtime.orbit_view(cam, v)
        views.append(v)
        cams.append(cam)
    return views, cams


def _surface_ray(rng, power, iters):
    """A ray from a camera on a sphere around the bulb that meets its surface: origin,
    unit direction, distance (an FP64 sphere trace on the host)."""

    def de(p):
        z, dr = list(p), 1.0
        for _ in range(iters):
            r = math.sqrt(sum(x * x for x in z))
            if r > 2.0:
                break
            th, ph = math.acos(max(-1.0, min(1.0, z[2] / r))) * power, math.atan2(z[1], z[0]) * power
            rp = r ** (power - 1.0)
            dr = rp * power * dr + 1.0
            z = [rp * r * math.sin(th) * math.cos(ph) + p[0], rp * r * math.sin(th) * math.sin(ph) + p[1],
                 rp * r * math.cos(th) + p[2]]
        r = math.sqrt(sum(x * x for x in z))
        return min(0.5 * math.log(max(r, 1e-6)) * r / dr, r)

    while True:
        org = _orbit_position(rng, 2.5)
        aim = [rng.uniform(-0.4, 0.4) - x for x in org]
        n = math.sqrt(sum(x * x for x in aim))
        d, t = [x / n for x in aim], 0.0
        for _ in range(4000):
            step = de([org[i] + d[i] * t for i in range(3)])
            if step < 1e-9 * t:
                return org, d, t
            t += step
            if t > 6.0:
                break


def _lite(view):
    return abi.make_lite(STOPS, LIGHTS)


def _rays(views):
    return sum(abi.rays_of(v) for v in views)


def prepare(case, seed):
    views, cams = _views(case, seed)
    n = _rays(views)
    kind = case["kind"]
    s = {"kind": kind, "ctx": _context(), "views": views, "opts": None}
    if kind in ("batch", "graph"):
        # the formats of the reference's targets: R32F depth, RGBA16F normal, trap, steps
        g = runtime.GBuffer.allocate(n, full=False)
        g.normal_half = torch.empty((n, 4), dtype=torch.float16, device="cuda")
        g.trap = torch.empty(n, dtype=torch.float32, device="cuda")
        g.steps = torch.empty(n, dtype=torch.int32, device="cuda")
        s["names"] = ("depth", "normal_half", "trap", "steps")
    elif kind == "diff":
        g = runtime.GBuffer.allocate(n, full=False)
        g.normal = torch.empty((n, 4), dtype=torch.float32, device="cuda")
        g.shade = torch.empty(n, dtype=torch.float32, device="cuda")
        g.depth64 = torch.empty(n, dtype=torch.float64, device="cuda")
        s["names"] = ("normal", "shade", "depth64")
        s["cams"], s["precision"], s["target"] = cams, case["precision"], _target(n, seed)
        if case["precision"] == 64:
            s["opts"] = runtime.make_opts(de_precision=64)
    else:
        g = runtime.GBuffer.allocate(n)
        s["names"] = ("depth", "normal", "trap", "steps", "iters", "shade", "shadow", "depth64", "evals")
        if kind == "closeup":
            s["opts"] = runtime.make_opts(de_precision=64)
        if kind == "lite":
            s["lites"] = [_lite(v) for v in views]
    s["g"] = g
    if kind == "graph":
        s["graph"] = s["ctx"].capture(views, g)
    return s


def _target(n, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return 0.3 + 0.5 * torch.rand(n, generator=gen, device="cuda")


def run(s):
    ctx, views, g = s["ctx"], s["views"], s["g"]
    if s["kind"] == "graph":
        s["graph"].launch()
    else:
        ctx.forward(views, g, s["opts"])
    out = {k: getattr(g, k) for k in s["names"]}
    if s["kind"] == "lite":
        out["rgba"] = ctx.shade_lite(views, s["lites"], g)
    if s["kind"] == "diff":
        dl = (g.shade - s["target"]) * (2.0 / g.shade.numel())
        if s["precision"] == 64:
            out["grad"], out["per_ray"] = ctx.backward(views, s["cams"], g, dl, param_idx=(0, 2), de_precision=64,
                                                       per_ray=True)
        else:
            out["grad"] = ctx.backward(views, s["cams"], g, dl, param_idx=(0, 2))
    return out


def work(case):
    """Bytes: the G-buffer written once (and read once where a later pass needs it).
    FLOPs: DE evaluations per ray, as these views need them, x iterations until the orbit
    escapes x about 70 operations per power step (transcendentals as one)."""
    kind = case["kind"]
    if kind in ("batch", "graph"):
        shape = random.Random(case["views"] * 1000 + case["max"])
        n = 0
        for _ in range(case["views"]):
            w, h = (int(round(math.exp(shape.uniform(math.log(case["min"]), math.log(case["max"]))))) for _ in range(2))
            n += w * h
        per, evals = 20, 18
    elif kind == "diff":
        n, evals = case["problems"] * case["side"] ** 2, 35 + 12
        per = 28 + 20 + (40 if case["precision"] == 64 else 0)
    else:
        n = case["w"] * case["h"] * case.get("spp", 1)
        per, evals = 52, {"view": 20, "lite": 20, "accel": 14, "closeup": 40}[kind]
        if kind == "lite":
            per += 16 + 28
        if kind == "accel":
            per += 6 * case["res"] ** 3 * 4 / n
    return {"bytes": float(n * per), "flops": float(n * evals * min(case["iters"], 5) * 70)}


# ---------------------------------------------------------------- FP64 restatement
F64 = torch.float64


def _t(x):
    return torch.as_tensor(x, dtype=F64, device="cuda")


def _step(z, dr, p, power, bail):
    r = (z[0] * z[0] + z[1] * z[1] + z[2] * z[2]).sqrt()
    go = ~(r > bail)
    th = torch.acos((z[2] / r).clamp(-1.0, 1.0)) * power
    ph = torch.atan2(z[1], z[0]) * power
    rp = r ** (power - 1.0)
    zr, st = rp * r, torch.sin(th)
    nz = (zr * (st * torch.cos(ph)) + p[0], zr * (st * torch.sin(ph)) + p[1], zr * torch.cos(th) + p[2])
    return tuple(torch.where(go, a, b) for a, b in zip(nz, z)), torch.where(go, rp * power * dr + 1.0, dr), go


def _de(p, q, trap=None):
    """DE at p (three tensors) for view parameters q; with a trap descriptor also the
    orbit trap (minimum over the iterations)."""
    z, dr = p, torch.ones_like(p[0])
    acc = torch.full_like(p[0], 1e6)
    for i in range(q["iters"]):
        z, dr, go = _step(z, dr, p, q["power"], q["bail"])
        if trap is not None:
            acc = torch.minimum(acc, _trap_distance(z, trap))
        if i % 3 == 2 and trap is None and not torch.is_grad_enabled() and not bool(go.any()):
            break
    r = (z[0] * z[0] + z[1] * z[1] + z[2] * z[2]).sqrt()
    d = torch.minimum(0.5 * torch.log(r.clamp_min(1e-6)) * r / dr.clamp_min(1e-6), r)
    return d if trap is None else (d, acc)


def _trap_distance(z, t):
    c = [z[i] - t["center"][i] for i in range(3)]
    if t["shape"] == abi.ND_TRAP_BOX:
        e = [c[i].abs() - t["box"][i] for i in range(3)]
        out = sum(x.clamp_min(0.0) ** 2 for x in e).sqrt()
        return (out + torch.maximum(e[0], torch.maximum(e[1], e[2])).clamp_max(0.0)).abs()
    n = (c[0] * c[0] + c[1] * c[1] + c[2] * c[2]).sqrt()
    return (n - t["radius"]).abs() if t["shape"] == abi.ND_TRAP_SPHERE else n


def _mix64(x):
    m = 0xFFFFFFFFFFFFFFFF
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return (x ^ (x >> np.uint64(31))) & np.uint64(m)


def _camera(v):
    """Per ray of view v: camera-plane coordinates and unit direction."""
    w, h, spp = v.width, v.height, v.spp
    idx = np.arange(spp * w * h, dtype=np.uint64)
    s, pix = idx // np.uint64(w * h), idx % np.uint64(w * h)
    px, py = pix % np.uint64(w), pix // np.uint64(w)
    jx = jy = 0.5
    if spp > 1:
        with np.errstate(over="ignore"):
            hash_ = _mix64(np.uint64(v.seed) ^ _mix64((s * np.uint64(h) + py) * np.uint64(w) + px))
        jx = ((hash_ & np.uint64(0xFFFFFFFF)) >> np.uint64(8)).astype(np.float64) / 16777216.0
        jy = (hash_ >> np.uint64(40)).astype(np.float64) / 16777216.0
    ux = _t((2.0 * (px.astype(np.float64) + jx) / w - 1.0) * (w / h))
    uy = _t(-(1.0 - 2.0 * (py.astype(np.float64) + jy) / h))
    d = [v.fwd[i] + v.right[i] * ux + v.up[i] * uy for i in range(3)]
    n = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt()
    return ux, uy, n, tuple(x / n for x in d)


class _Grid:
    """The accelerator's cascade of safe distances around a camera (placement in f32)."""

    def __init__(self, v, q):
        f = np.float32
        self.res, self.levels = v.accel_res // 4 * 4, v.accel_levels
        coarse = max(f(2.0) * f(v.max_dist) / f(self.res), f(1e-6))
        k = torch.arange(self.res, dtype=F64, device="cuda") + 0.5
        self.at, self.cell, grids = [], [], []
        for l in range(self.levels):
            cell = f(coarse / f(1 << (self.levels - 1 - l)))
            half = f(f(0.5) * f(self.res) * cell)
            at = [float(f(np.floor((f(v.cam_pos[a]) - half) / cell) * cell)) for a in range(3)]
            cell = float(cell)
            z, y, x = torch.meshgrid(at[2] + k * cell, at[1] + k * cell, at[0] + k * cell, indexing="ij")
            d = _de((x.reshape(-1), y.reshape(-1), z.reshape(-1)), q)
            grids.append((d - 0.5 * math.sqrt(3.0) * cell).clamp_min(0.0) * float(f(v.accel_safety)))
            self.at.append(at)
            self.cell.append(cell)
        self.grid = torch.cat(grids)

    def skip(self, p):
        out, open_ = torch.zeros_like(p[0]), torch.ones_like(p[0], dtype=torch.bool)
        for l in range(self.levels):
            c = [((p[a] - self.at[l][a]) / self.cell[l]).floor() for a in range(3)]
            inside = open_
            for x in c:
                inside = inside & (x >= 0) & (x < self.res)
            c = [x.clamp(0, self.res - 1).long() for x in c]
            i = ((l * self.res + c[2]) * self.res + c[1]) * self.res + c[0]
            out = torch.where(inside, self.grid[i], out)
            open_ = open_ & ~inside
        return out


def _params(v):
    return {"power": float(v.params[0]), "iters": int(v.params[1]), "bail": float(v.params[2])}


def _march(v, dirs, q):
    """Hit mask and distance of every ray (march_to sample by sample, rays in lockstep)."""
    n = dirs[0].numel()
    org = [v.cam_pos[i] for i in range(3)]
    hit, t_out = torch.zeros(n, dtype=torch.bool, device="cuda"), torch.zeros(n, dtype=F64, device="cuda")
    grid = _Grid(v, q) if v.accel_res > 0 else None
    refine, bisect = (v.refine_budget, 0) if v.march_verify else (0, v.refine_budget)
    foot = v.hq_footprint_px * 2.0 / v.height
    most = v.max_steps * (1 + refine) + bisect
    exact_hit = bool(v.flags & abi.ND_VIEW_EXACT_HIT)
    ids, d = torch.arange(n, device="cuda"), list(dirs)
    z = torch.zeros(n, dtype=F64, device="cuda")
    t, a, b = z, z, z
    i = torch.zeros(n, dtype=torch.int64, device="cuda")
    m, k = i, i
    no = torch.zeros(n, dtype=torch.bool, device="cuda")
    probing, bis, res, done = ~no, no, no, no

    def eps(x):
        return float(v.eps_coef) * x + float(v.eps_floor)

    turn = 0
    while ids.numel():
        if grid is not None:
            while True:
                s = grid.skip([org[j] + d[j] * t for j in range(3)])
                go = probing & ~done & (s > eps(t))
                if not bool(go.any()):
                    break
                a, t = torch.where(go, t, a), torch.where(go, t + s, t)
                i, m = i + go, m + go
                done = done | (go & ((t > v.max_dist) | (i >= v.max_steps) | (m >= most)))
        st = torch.where(probing, t, 0.5 * (a + b))
        de = _de(tuple(org[j] + d[j] * st for j in range(3)), q) * min(max(v.step_safety, 0.001), 1.0)
        live = ~done
        m = m + live
        below = de < eps(st)
        # in a bisection
        x = live & bis
        b = torch.where(x & below, st, b)
        a = torch.where(x & ~below, st, a)
        k = k + x
        stop = x & ((k >= bisect) | ((b - a <= eps(st)) if not exact_hit else no[: x.numel()]))
        got, at = stop, b
        done = done | (x & ~stop & (m >= most))
        # a sample under eps
        y = live & ~bis & below
        if bisect > 0:
            start = y & ((st > a) if exact_hit else (st - a > eps(st)))
            bis, probing = bis | start, probing & ~start
            b = torch.where(start, st, b)
            k = torch.where(start, 0, k)
            done = done | (start & (m >= most))
            y = y & ~start
        at = torch.where(y, st, at)
        got = got | y
        # a step
        w = live & ~(x | below)
        if not v.march_verify:
            a, t = torch.where(w, t, a), torch.where(w, t + de, t)
            i = i + w
            done = done | (w & ((t > v.max_dist) | (i >= v.max_steps) | (m >= most)))
        else:
            p1, p2 = w & probing, w & ~probing
            a, b = torch.where(p1, t, a), torch.where(p1, t + de, b)
            k = torch.where(p1, 0, k)
            res = res & ~p1
            safe = p2 & (de >= b - st)
            res = res | safe
            b = torch.where(p2 & ~safe, st, b)
            k = k + p2
            probing = probing & ~p1
            adv = w & (res | (k >= refine))
            if v.high_quality and refine > 0:
                b = torch.where(adv & ~res, torch.minimum(b, a + t.clamp_min(1.0) * foot), b)
            t = torch.where(adv, b, t)
            i = i + adv
            over = adv & ((t > v.max_dist) | (i >= v.max_steps))
            probing = probing | adv
            done = done | over | (w & (m >= most))
        if bool(got.any()):
            hit[ids[got]] = True
            t_out[ids[got]] = at[got]
            done = done | got
        turn += 1
        if turn % 8 == 0 or bool(done.all()):
            keep = ~done
            if int(keep.sum()) < 0.8 * keep.numel():
                ids, t, a, b, i, m, k = (u[keep] for u in (ids, t, a, b, i, m, k))
                probing, bis, res, done = (u[keep] for u in (probing, bis, res, done))
                d = [u[keep] for u in d]
                no = no[: ids.numel()]
    return hit, t_out


def _central(v, p, h, q):
    """The central-difference vector of the DE at p."""
    g = []
    for j in range(3):
        e = [h if u == j else 0.0 for u in range(3)]
        g.append(_de(tuple(p[u] + e[u] for u in range(3)), q) - _de(tuple(p[u] - e[u] for u in range(3)), q))
    return g


def _normal(v, p, t, q):
    eps = float(v.eps_coef) * t + float(v.eps_floor)
    if v.normal_mode == abi.ND_NORMAL_CENTRAL:
        g = _central(v, p, float(v.normal_h_coef) * t if v.normal_h_coef > 0 else eps, q)
    else:
        g = [torch.zeros_like(t)] * 3
        for k in ((1, -1, -1), (-1, -1, 1), (-1, 1, -1), (1, 1, 1)):
            d = _de(tuple(p[u] + k[u] * eps for u in range(3)), q)
            g = [g[u] + k[u] * d for u in range(3)]
    l = sum(x * x for x in g).sqrt()
    return [x / l for x in g]


def _unit(x):
    n = math.sqrt(sum(float(u) * float(u) for u in x))
    return [float(u) / n for u in x]


def _shadow(v, p, n, q):
    so = [p[j] + 0.004 * n[j] for j in range(3)]
    light = _unit(v.light_dir)
    vis = torch.ones_like(p[0])
    ids, a, res = torch.arange(vis.numel(), device="cuda"), torch.full_like(vis, 0.004), torch.ones_like(vis)
    for _ in range(min(v.max_steps, 40)):
        d = _de(tuple(so[j] + light[j] * a for j in range(3)), q)
        dark = d < 0.0005
        res = torch.minimum(res, v.shadow_k * d / a)
        a = a + d.clamp_min(0.001)
        out = dark | (a >= 2.0 * v.max_dist)
        vis[ids] = torch.where(dark, 0.0, res.clamp(0.0, 1.0))
        ids, a, res = ids[~out], a[~out], res[~out]
        so = [x[~out] for x in so]
        if not ids.numel():
            break
    return vis


def _trap_of(v):
    return {"shape": v.trap.shape, "center": list(v.trap.center), "box": list(v.trap.box), "radius": float(v.trap.radius)}


def _lambert(v, d, n, vis):
    if v.shadow or any(v.light_dir):
        key = _unit(v.light_dir)
    else:
        r, u = _unit(v.right), _unit(v.up)
        key = [-d[j] + 0.45 * u[j] - 0.35 * r[j] for j in range(3)]
        l = sum(x * x for x in key).sqrt()
        key = [x / l for x in key]
    return 0.18 + 0.82 * sum(n[j] * key[j] for j in range(3)).clamp_min(0.0) * vis


def _strip(t, x):
    x = x / max(float(t.span), 1e-4) + float(t.offset)
    if t.repeat == 1:
        return x - x.floor()
    if t.repeat == 2:
        return 1.0 - ((x * 0.5 - (x * 0.5).floor()) * 2.0 - 1.0).abs()
    return x.clamp(0.0, 1.0)


def _shade_lite(v, d, p, t, n, trap, q):
    x = _strip(v.trap, trap)
    rows = [list(c) + [g, ior] for c, _, g, ior in STOPS]
    at = [s for _, s, _, _ in STOPS]
    mat = []
    for j in range(5):
        u = torch.full_like(x, rows[-1][j])
        for k in range(len(rows) - 2, -1, -1):
            f = (x - at[k]) / (at[k + 1] - at[k])
            u = torch.where(x <= at[k + 1], rows[k][j] * (1.0 - f) + rows[k + 1][j] * f, u)
        mat.append(torch.where(x <= at[0], rows[0][j], u))
    radius = (0.04 * t).clamp(0.003, 0.25)
    occ, weight = torch.zeros_like(t), 1.0
    for k in range(5):
        step = radius * (0.2 + 0.2 * k)
        occ = occ + (step - _de(tuple(p[j] + n[j] * step for j in range(3)), q)).clamp_min(0.0) * weight
        weight *= 0.6
    amb = 0.15 * (1.0 - 2.0 * occ / radius).clamp(0.0, 1.0)
    ior = mat[4].clamp_min(1.0)
    r0 = ((1.0 - ior) / (1.0 + ior)) ** 2
    fres = r0 + (1.0 - r0) * (1.0 - sum(d[j] * n[j] for j in range(3)).abs()).clamp(0.0, 1.0) ** 5
    power = 4.0 + 124.0 * mat[3].clamp(0.0, 1.0)
    diff, spec = [amb] * 3, [torch.zeros_like(t)] * 3
    for kind, where, rgb, bright in LIGHTS:
        c = [x * bright for x in rgb]
        if kind == abi.ND_LIGHT_POINT:
            l = [where[j] - p[j] for j in range(3)]
            dist = sum(x * x for x in l).sqrt()
            l = [x / dist.clamp_min(1e-4) for x in l]
            c = [x / (dist * dist).clamp_min(0.01) for x in c]
        else:
            l = [torch.full_like(t, x) for x in _unit(where)]
        nl = sum(n[j] * l[j] for j in range(3)).clamp_min(0.0)
        h = [l[j] - d[j] for j in range(3)]
        hl = sum(x * x for x in h).sqrt()
        sp = sum(n[j] * h[j] / hl for j in range(3)).clamp_min(0.0) ** power * mat[3] * (nl > 0)
        diff = [diff[j] + c[j] * nl for j in range(3)]
        spec = [spec[j] + c[j] * sp for j in range(3)]
    return [(1.0 - fres) * (mat[j] * diff[j] + spec[j]) for j in range(3)]


def _pose(cam, x):
    """Origin, forward, right and up of an orbit camera for x = (yaw, pitch, dist)."""
    yaw, pitch, dist = x
    off = torch.stack([torch.cos(pitch) * torch.sin(yaw), torch.sin(pitch), -torch.cos(pitch) * torch.cos(yaw)])
    org = _t(list(cam.target)) + dist * off
    f = _t(list(cam.target)) - org
    f = f / f.norm()
    r = torch.linalg.cross(f, _t(list(cam.world_up)))
    r = r / r.norm()
    u = torch.linalg.cross(r, f)
    sc = math.tan(math.radians(cam.fov_y_deg) * 0.5)
    return torch.stack([org, f, r * sc, u / u.norm() * sc])


def _de_tangent(p, dp, q, dpower):
    """DE at p and its derivative along (dp, dpower) (forward differentiation by torch)."""

    def f(x, y, z, power):
        return _de((x, y, z), {**q, "power": power})

    power = torch.full_like(p[0], q["power"])
    with torch.enable_grad():
        return torch.func.jvp(f, (*p, power), (*dp, torch.full_like(power, dpower)))


def _jacobian(v, cam, ux, uy, wn, d, t, q, n, precision):
    """d shade / d (power, bailout, yaw, pitch, dist) at hits: implicit differentiation of
    DE(p) = eps(t) through the central-difference normal."""
    J = torch.autograd.functional.jacobian(lambda x: _pose(cam, x), _t([cam.yaw, cam.pitch, cam.dist]))  # 4 x 3 x 3
    p = [v.cam_pos[j] + d[j] * t for j in range(3)]
    zero = torch.zeros_like(t)
    g, value = [], None
    for j in range(3):
        value, x = _de_tangent(p, [zero + float(u == j) for u in range(3)], q, 0.0)
        g.append(x)
    coef, eps = float(v.eps_coef), float(v.eps_coef) * t + float(v.eps_floor)
    root = (value - eps).abs() <= (1e-6 if precision == 64 else 1e-2) * eps
    denom = sum(g[j] * d[j] for j in range(3)) - coef
    hc = float(v.normal_h_coef)
    h = hc * t
    D = _central(v, p, h, q)
    Dn = sum(x * x for x in D).sqrt()
    light = _unit(v.light_dir)
    n = [x / Dn for x in D]
    ok = root & (sum(n[j] * light[j] for j in range(3)) > 0) & (denom != 0)
    cols = []
    for k in range(5):
        if k < 2:
            tan, seed = [zero] * 3, 1.0 if k == 0 else 0.0
        else:
            j = k - 2
            dw = [J[1, u, j] + ux * J[2, u, j] + uy * J[3, u, j] for u in range(3)]
            par = sum(d[u] * dw[u] for u in range(3))
            tan, seed = [J[0, u, j] + t * (dw[u] - d[u] * par) / wn for u in range(3)], 0.0
        if k == 1:  # the escape radius enters through a comparison only
            cols.append(zero)
            continue
        dt = -_de_tangent(p, tan, q, seed)[1] / denom
        dp, dh = [tan[u] + dt * d[u] for u in range(3)], hc * dt
        dD = []
        for j in range(3):
            hi = _de_tangent([p[u] + (h if u == j else 0.0) for u in range(3)],
                             [dp[u] + (dh if u == j else 0.0) for u in range(3)], q, seed)[1]
            lo = _de_tangent([p[u] - (h if u == j else 0.0) for u in range(3)],
                             [dp[u] - (dh if u == j else 0.0) for u in range(3)], q, seed)[1]
            dD.append(hi - lo)
        nd = sum(n[u] * dD[u] for u in range(3))
        cols.append(0.82 * sum(light[u] * (dD[u] - n[u] * nd) / Dn for u in range(3)))
    return torch.where(ok[:, None], torch.stack(cols, 1), torch.zeros((), dtype=F64, device="cuda"))


def exact(case, seed):
    views, cams = _views(case, seed)
    outs = []
    with torch.no_grad():
        for vi, v in enumerate(views):
            q = _params(v)
            ux, uy, wn, dirs = _camera(v)
            hit, t = _march(v, dirs, q)
            rays = t.numel()
            hd = [x[hit] for x in dirs]
            ht = t[hit]
            p = [v.cam_pos[j] + hd[j] * ht for j in range(3)]
            n = _normal(v, p, ht, q)
            vis = _shadow(v, p, n, q) if v.shadow else torch.ones_like(ht)

            def put(x, miss=0.0):
                full = torch.full((rays,), miss, dtype=F64, device="cuda")
                full[hit] = x
                return full

            o = {"depth": put(ht), "normal": torch.stack([put(x) for x in n] + [hit.to(F64)], 1),
                 "shade": put(_lambert(v, hd, n, vis)), "shadow": put(vis, 1.0)}
            o["depth64"], o["normal_half"] = o["depth"], o["normal"]
            if case["kind"] != "diff":
                trap = _de(tuple(p), q, _trap_of(v))[1]
                o["trap"] = put(trap)
            if case["kind"] == "lite":
                rgb = _shade_lite(v, hd, p, ht, n, trap, q)
                back = list(_lite(v).background)
                o["rgba"] = torch.stack([put(x, back[j]) for j, x in enumerate(rgb)] + [hit.to(F64)], 1)
            if case["kind"] == "diff":
                jac = torch.zeros((rays, 5), dtype=F64, device="cuda")
                jac[hit] = _jacobian(v, cams[vi], ux[hit], uy[hit], wn[hit], hd, ht, q, n, case["precision"])
                o["per_ray"] = jac
            outs.append(o)
        cat = {k: torch.cat([o[k] for o in outs]) for k in outs[0]}
        if case["kind"] in ("batch", "graph"):
            return {"depth": cat["depth"], "normal_half": cat["normal_half"], "trap": cat["trap"], "steps": None}
        if case["kind"] == "diff":
            total = cat["shade"].numel()
            dl = (cat["shade"] - _target(total, seed).to(F64)) * (2.0 / total)
            rays = case["side"] ** 2
            grad = torch.stack([(dl[i * rays:(i + 1) * rays, None] * outs[i]["per_ray"]).sum(0) for i in range(len(views))])
            r = {k: cat[k] for k in ("normal", "shade", "depth64")}
            # a few hits on the jumps of a non-integer power carry most of a Jacobian's
            # norm, and rounding decides which hits those are (all of them for an FP32 DE)
            if case["precision"] == 32:
                return {**r, "grad": None}
            return {**r, "grad": grad, "per_ray": None}
        r = {k: cat[k] for k in ("depth", "normal", "trap", "shade", "shadow", "depth64")}
        r.update(steps=None, iters=None, evals=None)
        if case["kind"] == "lite":
            r["rgba"] = cat["rgba"]
        return r
