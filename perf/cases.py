"""Workloads of the framework as its users run them: batches of rays traced
against meshes and scenes, reference-mode and path-traced renders, the path
guide's training gradient.  Each case goes through the public Python
interface (vermeer_gb300.Context), which is the C ABI's calls one to one.

A program keeps one context with its scene loaded and calls it many times;
prepare() builds that (meshes and their accelerators included) and run() is
one call.  Device-resident rays and hits live on one stream, which the
contexts and torch share, as a program that mixes both would do."""
import math

import numpy as np
import torch

import vermeer_gb300 as vg
from vermeer_gb300 import scenes

_STREAM = None


def _stream():
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def listed():
    return [
        # A picking or probing call of an interactive program: a handful of rays, where latency is all.
        dict(name="mesh_closest_small", kind="mesh", tris=1024, rays=1000, edge=0.05, shadow=False, coherent=False),
        # A visibility pass of ragged size: camera-like rays with a finite reach, hit or miss wanted.
        dict(name="mesh_any_ragged", kind="mesh", tris=200003, rays=300007, edge=0.005, shadow=True, coherent=True),
        # The raw-traversal benchmark: a million triangles, four million incoherent rays.
        dict(name="mesh_closest_large", kind="mesh", tris=1048576, rays=4194304, edge=0.005, shadow=False,
             coherent=False),
        # Motion blur: two-key motion, every ray at its own time.
        dict(name="mesh_motion", kind="motion", tris=100000, rays=262147, edge=0.005, velocity=0.05),
        # A two-level scene of many meshes (the sphere grid), rays from all over it.
        dict(name="scene_closest", kind="scene", per_side=6, subdiv=24, rays=1000003, shadow=False),
        # Rays and hits in host memory, as a host renderer's batches are.
        dict(name="mesh_closest_host", kind="host", tris=20000, rays=300000, edge=0.01),
        # core.Render, reference mode, the small room as configured.
        dict(name="render_ref_room", kind="ref", tris=16384, res=256, iters=16, light_samples=1, f32=False),
        # The extended path tracer's full image: displaced spheres, diffuse + GGX, quad lights, environment.
        dict(name="path_grid", kind="path_grid", per_side=8, subdiv=32, width=1920, height=1080, iters=4, depth=8),
        # A preview tile of the room with every light kind and lobe: short queues, launch latency.
        dict(name="path_room_small", kind="path_room", tris=4096, width=64, height=48, iters=1, depth=4),
        # A frame of the slit-light room rendered with the path guide.
        dict(name="path_guided", kind="path_guided", tris=50000, width=512, height=512, iters=2, depth=8,
             guide_depth=2),
        # Many small one-mesh renders, half of them with motion, in one call.
        dict(name="path_jobs", kind="path_jobs", jobs=16, tri_max=50000, size=128, iters=8, depth=5),
        # One batch of the guide's training: forward, loss and backward to every weight.
        dict(name="guide_gradient", kind="guide", rows=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mesh", "mesh", "motion", "scene", "host", "ref", "path_grid", "path_room", "path_guided",
                       "path_jobs", "guide"])
    if kind == "mesh":
        tris = _log(rng, 64, 1000000)
        return dict(kind=kind, tris=tris, rays=_log(rng, 257, 4000000), edge=round(0.5 * tris ** (-1 / 3), 5),
                    shadow=rng.random() < 0.5, coherent=rng.random() < 0.5)
    if kind == "motion":
        return dict(kind=kind, tris=_log(rng, 1000, 200000), rays=_log(rng, 1000, 500000), edge=0.005,
                    velocity=round(rng.uniform(0.01, 0.08), 3))
    if kind == "scene":
        return dict(kind=kind, per_side=rng.randint(2, 7), subdiv=rng.randint(8, 28), rays=_log(rng, 5000, 2000000),
                    shadow=rng.random() < 0.5)
    if kind == "host":
        return dict(kind=kind, tris=_log(rng, 500, 30000), rays=_log(rng, 100, 500000), edge=0.01)
    if kind == "ref":
        return dict(kind=kind, tris=_log(rng, 500, 30000), res=rng.randint(33, 300), iters=rng.randint(1, 12),
                    light_samples=rng.randint(0, 2), f32=rng.random() < 0.3)
    if kind == "path_grid":
        return dict(kind=kind, per_side=rng.randint(2, 7), subdiv=rng.randint(8, 32), width=rng.randint(200, 1920),
                    height=rng.randint(150, 1080), iters=rng.randint(1, 4), depth=rng.randint(2, 8))
    if kind == "path_room":
        return dict(kind=kind, tris=_log(rng, 500, 20000), width=rng.randint(17, 400), height=rng.randint(17, 300),
                    iters=rng.randint(1, 6), depth=rng.randint(1, 8))
    if kind == "path_guided":
        return dict(kind=kind, tris=_log(rng, 2000, 60000), width=rng.randint(64, 512), height=rng.randint(64, 512),
                    iters=rng.randint(1, 2), depth=rng.randint(2, 8), guide_depth=rng.randint(1, 2))
    if kind == "path_jobs":
        return dict(kind=kind, jobs=rng.randint(2, 16), tri_max=_log(rng, 2000, 50000), size=rng.randint(32, 128),
                    iters=rng.randint(1, 8), depth=rng.randint(1, 5))
    return dict(kind="guide", rows=_log(rng, 1000, 100000))


# ------------------------------------------------------------------ inputs ---
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _sphere(g, n):
    d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True).clamp_min(1e-12)


def _soup(g, n, edge, velocity=0.0):
    """A soup in the unit cube: centroids uniform, vertices at centroid + edge * (a direction uniform on the
    sphere); with a velocity, a second key moved by a vector drawn in a ball of that radius per triangle."""
    c = torch.rand((n, 1, 3), generator=g, device="cuda", dtype=torch.float64)
    v = (c + edge * _sphere(g, 3 * n).reshape(n, 3, 3)).float()
    if velocity == 0.0:
        return v.reshape(-1, 3)
    r = velocity * torch.rand((n, 1), generator=g, device="cuda", dtype=torch.float64) ** (1 / 3)
    w = (v.double() + (_sphere(g, n) * r)[:, None, :]).float()
    return torch.cat([v.reshape(-1, 3), w.reshape(-1, 3)])


def _rays(g, n, coherent=False, tmax=math.inf, lo=(0.0, 0.0, 0.0), hi=(1.0, 1.0, 1.0), times=False):
    """[8, n]: origins uniform in a box and directions uniform on the sphere, or (coherent) a pinhole's rays in
    scanline order through a square image."""
    r = torch.empty((8, n), device="cuda", dtype=torch.float32)
    if coherent:
        eye = torch.tensor([0.5, 0.5, -1.2], device="cuda", dtype=torch.float64)
        eye = eye + 0.05 * torch.randn(3, generator=g, device="cuda", dtype=torch.float64)
        side = math.isqrt(n - 1) + 1
        k = torch.arange(n, device="cuda")
        sx = ((k % side).double() + 0.5) / side * 2 - 1
        sy = 1 - ((k // side).double() + 0.5) / side * 2
        d = torch.stack([sx, sy, torch.full_like(sx, 2.75)], dim=1) * 0.36
        r[0:3] = eye.float()[:, None]
        r[3:6] = (d / d.norm(dim=1, keepdim=True)).T.float()
    else:
        a = torch.tensor(lo, device="cuda", dtype=torch.float64)
        b = torch.tensor(hi, device="cuda", dtype=torch.float64)
        r[0:3] = (a + (b - a) * torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)).T.float()
        r[3:6] = _sphere(g, n).T.float()
    r[6] = tmax
    r[7] = torch.rand(n, generator=g, device="cuda") if times else 0.0
    return r


def _index(n):
    return np.arange(3 * n, dtype=np.uint32)


def _guide_rows(g, n):
    def unit():
        return _sphere(g, n).float().cpu().numpy()
    pos = (torch.rand((n, 3), generator=g, device="cuda") * 2 - 1).cpu().numpy()
    nrm, wo, om = unit(), unit(), unit()
    weight = (torch.rand(n, generator=g, device="cuda") + 0.25).cpu().numpy()
    pdf = np.maximum((nrm * om).sum(1), 0).astype(np.float32) / np.float32(math.pi)
    return pos, nrm, wo, om, weight, pdf


_GUIDE_SHAPES = [(64, 80), (64, 64), (64, 64), (64, 64), (41, 64)]


def _guide_weights(seed):
    g = torch.Generator()
    g.manual_seed(seed)
    w = [torch.randn(a * b, generator=g) * math.sqrt(2.0 / b) for a, b in _GUIDE_SHAPES]
    w[4] *= 0.3
    return torch.cat(w).numpy()


def _inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "mesh":
        v = _soup(g, case["tris"], case["edge"])
        return v, _rays(g, case["rays"], case["coherent"], tmax=2.0 if case["shadow"] else math.inf)
    if case["kind"] == "motion":
        v = _soup(g, case["tris"], case["edge"], case["velocity"])
        return v, _rays(g, case["rays"], times=True)
    if case["kind"] == "host":
        v = _soup(g, case["tris"], case["edge"])
        return v, _rays(g, case["rays"])
    raise ValueError(case["kind"])


def prepare(case, seed):
    kind = case["kind"]
    torch.cuda.current_stream().synchronize()
    ctx = vg.Context(0)
    s = dict(case=case, ctx=ctx, seed=seed)
    if kind in ("mesh", "motion", "host"):
        v, rays = _inputs(case, seed)
        s["geom"] = ctx.mesh_build(v.cpu().numpy(), _index(case["tris"]), keys=2 if kind == "motion" else 1,
                                   motion_mode=vg.MOTION_FIXED if kind == "motion" else vg.MOTION_FAITHFUL)
        s["rays"] = rays.T.contiguous().cpu().numpy() if kind == "host" else rays
    elif kind in ("scene", "path_grid"):
        w, h = case.get("width", 1280), case.get("height", 720)
        ctx.load_scene(scenes.sphere_grid(case["per_side"], case["subdiv"], seed=3 + seed % 997, width=w, height=h))
        if kind == "scene":
            e = case["per_side"] / 2.0 + 1.0
            s["rays"] = _rays(_gen(seed), case["rays"], tmax=4.0 if case["shadow"] else math.inf,
                              lo=(-e, 0.01, -e), hi=(e, 3.0, e))
    elif kind == "ref":
        ctx.load_scene(scenes.small_room(case["tris"], seed=1 + seed % 997, light_samples=case["light_samples"]))
    elif kind == "path_room":
        ctx.load_scene(scenes.small_room_ext(case["tris"], seed=1 + seed % 997))
    elif kind == "path_guided":
        ctx.load_scene(scenes.slit_room(case["tris"], seed=5 + seed % 997, width=case["width"],
                                        height=case["height"]))
        ctx.guide_set_weights(_guide_weights(seed))
    elif kind == "path_jobs":
        bj = scenes.batched_jobs(case["jobs"], seed=4 + seed % 997, width=case["size"], height=case["size"], lo=1000,
                                 hi=case["tri_max"])
        ids = [ctx.mesh_build(m["verts"], m["idxp"], keys=m.get("keys", 1), motion_mode=m.get("motion_mode", 0))
               for m in bj["meshes"]]
        ctx.set_shaders(bj["shaders"])
        for k in ids:
            ctx.mesh_set_shading(k, [0])
        ctx.set_env_light(bj["env"])
        s["jobs"] = [dict(geom=k, width=bj["width"], height=bj["height"], camera=c)
                     for k, c in zip(ids, bj["cameras"])]
    else:
        ctx.guide_set_weights(_guide_weights(seed))
        s["rows"] = _guide_rows(_gen(seed), case["rows"])
    if kind in ("mesh", "motion", "scene"):
        ctx.set_stream(_stream().cuda_stream)
    return s


_LO, _HI = np.full(3, -1, np.float32), np.full(3, 1, np.float32)


def run(state):
    c, ctx, kind = state["case"], state["ctx"], state["case"]["kind"]
    if kind in ("mesh", "motion", "host"):
        with torch.cuda.stream(_stream()):
            r = ctx.trace_mesh(state["geom"], state["rays"], shadow=c.get("shadow", False))
        return {k: r[k] for k in ("prim", "t", "u", "v", "w")}
    if kind == "scene":
        with torch.cuda.stream(_stream()):
            r = ctx.trace_scene(state["rays"], shadow=c["shadow"])
        return {k: r[k] for k in ("prim", "geom", "t", "u", "v", "w")}
    if kind == "ref":
        return ctx.render(c["res"], c["res"], 0, c["iters"], state["seed"], f32=c["f32"])[0]
    if kind == "path_jobs":
        return ctx.render_path_jobs(state["jobs"], 0, c["iters"], state["seed"], max_depth=c["depth"])[0]
    if kind == "guide":
        pos, nrm, wo, om, weight, pdf = state["rows"]
        grad, loss = ctx.guide_gradient(pos, nrm, wo, om, weight, _LO, _HI, bsdf_pdf=pdf)
        return {"grad": grad.astype(np.float32), "loss": np.float32(loss)}
    more = dict(guided=True, guide_depth=c["guide_depth"]) if kind == "path_guided" else {}
    return ctx.render_path(c["width"], c["height"], 0, c["iters"], state["seed"], max_depth=c["depth"], **more)[0]


def work(case):
    """Bytes: inputs once, outputs once.  Operations: 32 box tests of 20 and 16 triangle tests of 60 a ray (about the
    least that finds a hit in these trees); a path is taken as three vertices of two rays."""
    kind = case["kind"]
    ray = 32 * 20 + 16 * 60
    if kind in ("mesh", "motion", "host"):
        keys = 2 if kind == "motion" else 1
        return {"bytes": case["rays"] * 52 + case["tris"] * 36 * keys, "flops": case["rays"] * ray}
    grid = case.get("per_side", 0) ** 2 * 8 * case.get("subdiv", 0) ** 2
    if kind == "scene":
        return {"bytes": case["rays"] * 56 + grid * 36, "flops": case["rays"] * ray}
    if kind == "guide":
        n = 20032
        return {"bytes": case["rows"] * 56 + n * 8, "flops": case["rows"] * n * 6}
    if kind == "path_jobs":
        pixels, tris = case["jobs"] * case["size"] ** 2, case["jobs"] * case["tri_max"] // 4
    elif kind == "ref":
        pixels, tris = case["res"] ** 2, case["tris"]
    else:
        pixels, tris = case["width"] * case["height"], case.get("tris", grid)
    return {"bytes": pixels * 24 + tris * 36, "flops": pixels * case["iters"] * 6 * ray}


# ------------------------------------------------------- 64-bit references ---
def _closest(v0, v1, rays):
    """The nearest hit of each ray by testing every triangle in float64 (v1: the second key of moving vertices)."""
    n = rays.shape[1]
    o, d, tm, time = rays[0:3].T.double(), rays[3:6].T.double(), rays[6].double(), rays[7].double()
    T = v0.shape[0]
    best = [tm.clone()] + [torch.zeros_like(tm) for _ in range(3)]
    step = max(1, 120_000_000 // max(1, T))
    for a in range(0, n, step):
        b = min(n, a + step)
        oo, dd = o[a:b], d[a:b]
        m = b - a
        if v1 is None:
            A, e1, e2 = v0[:, 0], v0[:, 1] - v0[:, 0], v0[:, 2] - v0[:, 0]
            nrm = torch.linalg.cross(e1, e2)
            q1, q2 = torch.linalg.cross(e2, A), torch.linalg.cross(A, e1)
            # triple products as matrix products: with c = o x d,
            # det = d.n, t = (A - o).n / det, and the barycentrics from d.(e x A) and c.e
            c = torch.linalg.cross(oo, dd)
            det = dd @ nrm.T
            tt = ((A * nrm).sum(1)[None, :] - oo @ nrm.T) / det
            v = (dd @ q1.T - c @ e2.T) / det
            w = (dd @ q2.T + c @ e1.T) / det
        else:
            s = time[a:b, None, None]
            tri = [(1 - s) * v0[None, :, k] + s * v1[None, :, k] for k in range(3)]
            A, e1, e2 = tri[0], tri[1] - tri[0], tri[2] - tri[0]
            nrm = torch.linalg.cross(e1, e2)
            det = (nrm * dd[:, None]).sum(2)
            r = A - oo[:, None]
            tt = (r * nrm).sum(2) / det
            x = torch.linalg.cross(r, dd[:, None].expand_as(r))
            v = (x * e2).sum(2) / det
            w = -(x * e1).sum(2) / det
        u = 1 - v - w
        tt = torch.where((u >= 0) & (v >= 0) & (w >= 0) & (tt > 0) & (det != 0), tt, math.inf)
        t, i = tt.min(1)
        hit = t < best[0][a:b]
        k = torch.arange(m, device=rays.device)
        best[0][a:b] = torch.where(hit, t, best[0][a:b])
        for q, f in zip(best[1:], (u, v, w)):
            q[a:b] = torch.where(hit, f[k, i], q[a:b])
    return best


def _guide_loss(case, seed):
    pos, nrm, wo, om, weight, pdf = (torch.from_numpy(a).cuda().double() for a in _guide_rows(_gen(seed), case["rows"]))
    w = torch.from_numpy(_guide_weights(seed)).cuda().double().requires_grad_(True)
    q = (pos + 1) / 2
    ang = math.pi * q[:, :, None] * (2.0 ** torch.arange(12, device="cuda", dtype=torch.float64))
    enc = torch.stack([torch.sin(ang), torch.cos(ang)], dim=3).reshape(-1, 72)
    one = torch.ones_like(weight)[:, None]
    x = torch.cat([enc, nrm, wo, one, 0 * one], dim=1)
    at = 0
    for k, (a, b) in enumerate(_GUIDE_SHAPES):
        x = x @ w[at:at + a * b].reshape(a, b).T
        at += a * b
        if k < 4:
            x = torch.relu(x)
    o = x[:, :40].reshape(-1, 8, 5)
    mu = o[:, :, :3] / o[:, :, :3].norm(dim=2, keepdim=True).clamp_min(1e-6)
    kap = torch.exp(o[:, :, 3].clamp(-4.6, 6.9))
    vmf = kap / (2 * math.pi * -torch.expm1(-2 * kap)) * torch.exp(kap * ((mu * om[:, None]).sum(2) - 1))
    p = (torch.softmax(o[:, :, 4], dim=1) * vmf).sum(1)
    alpha = 0.9 * torch.sigmoid(x[:, 40])
    full = -(weight * torch.log(alpha * p + (1 - alpha) * pdf)).sum()
    # the lobes descend the guide's own density, the selection the mixture's with the guide's density held
    goal = -(weight * torch.log(p)).sum() - (weight * torch.log(alpha * p.detach() + (1 - alpha) * pdf)).sum()
    goal.backward()
    return {"grad": w.grad, "loss": full.detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "guide":
        return _guide_loss(case, seed)
    # which triangle stops a shadow ray is the traversal's choice, and images are sums over thousands of random
    # decisions: neither has a value of its own in 64 bits
    if kind not in ("mesh", "motion", "host") or case.get("shadow"):
        return None
    cost = case["tris"] * case["rays"] * (8 if kind == "motion" else 1)
    if cost > 2.2e11:
        return None
    v, rays = _inputs(case, seed)
    v = v.double().reshape(2 if kind == "motion" else 1, -1, 3, 3)
    t, a, b, c = _closest(v[0], v[1] if kind == "motion" else None, rays)
    return {"prim": None, "t": t, "u": a, "v": b, "w": c}
