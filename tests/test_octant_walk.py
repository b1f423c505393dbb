"""The octant copies of the nodes (ONode) against the node-by-node kernel.

The while-while kernels walk per-octant copies whose children are in push
order and whose planes are near/far; the step-scheduled kernel (tuning
kernel 0) walks the nodes themselves.  Both must give the same bits for every
ray and every box an upload may hold: directions with zero, negative zero,
infinite and NaN components, boxes out of order, with NaN or infinite planes,
empty children, one key or several, finite and infinite reach.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OUT = ("prim", "t", "u", "v", "w")


def _rays(n, seed):
    from vermeer_gb300 import scenes
    r = scenes.incoherent_rays(n, seed)
    d = r[:, 3:6]
    d[0::16, 0] = 0.0
    d[1::16, 1] = -0.0
    d[2::16, 2] = 0.0
    d[3::16, :2] = 0.0
    d[4::16] = (0.0, -1.0, -0.0)
    d[5::64, 0] = np.inf
    d[6::64, 1] = np.nan
    d[7::64, 2] = 1e-42
    r[8::64, 0] = np.inf
    r[9::64, 3:6] *= 1e20
    r[10::16, 6] = 0.3
    r[11::64, 6] = np.nan
    r[12::64, 6] = -1.0
    r[:, 7] = scenes.uniform(seed, n, 77).astype(np.float32)
    r[13::16, 7] = 0.0
    r[14::16, 7] = 1.0
    return r


def _spoil(boxes, kind):
    b = boxes.reshape(-1, 24)
    if kind == "swapped":
        b[::3, [0, 12]] = b[::3, [12, 0]]
        b[1::5, [6, 18]] = b[1::5, [18, 6]]
    elif kind == "nan":
        b[::4, 3] = np.nan
        b[1::4, 14] = np.nan
        b[2::7] = np.nan
    elif kind == "inf":
        b[::3, 0:4] = -np.inf
        b[::3, 12:16] = np.inf


@pytest.mark.parametrize("kind", ["clean", "swapped", "nan", "inf"])
@pytest.mark.parametrize("keys", [1, 2, 3])
@pytest.mark.parametrize("tris", [1, 3, 17, 1500])
def test_octant_copies_equal_the_nodes(ctx, kind, keys, tris):
    from vermeer_gb300 import scenes
    v, ip = scenes.triangle_soup(tris, 11, edge=0.2 if tris < 100 else 0.06)
    if keys > 1:
        vs = [v + np.float32(0.1 * k) * scenes.unit_sphere(5 + k, v.shape[0], 3).astype(np.float32)
              for k in range(keys)]
        v = np.concatenate(vs).astype(np.float32)
    g = ctx.mesh_build(v, ip, keys=keys, motion_mode=1)
    if kind != "clean":
        e = ctx.mesh_export(g)
        if keys == 1:
            nodes = e["nodes"].copy()
            boxes = np.ascontiguousarray(nodes["boxes"])
            _spoil(boxes, kind)
            nodes["boxes"] = boxes
            g = ctx.mesh_upload(v, e["idxp"], e["accel_idx"], nodes=nodes, bounds=e["bounds"])
        else:
            boxes = e["mboxes"].copy()
            _spoil(boxes, kind)
            g = ctx.mesh_upload(v, e["idxp"], e["accel_idx"], mnodes=e["mnodes"], mboxes=boxes, bounds=e["bounds"],
                                keys=keys, motion_mode=1)
    rays = _rays(4099, 3)
    try:
        for shadow in (False, True):
            got = {}
            for k in (0, 13, 45):
                ctx.set_tuning(kernel=k)
                got[k] = ctx.trace_mesh(g, rays, shadow=shadow)
            assert (got[0]["prim"] >= 0).any() or kind == "nan" or tris < 100
            for k in (13, 45):
                for o in OUT:
                    a, b = got[k][o], got[0][o]
                    a, b = (x.view(np.uint32) if x.dtype == np.float32 else x for x in (a, b))
                    assert np.array_equal(a, b), (o, k, shadow)
    finally:
        ctx.set_tuning()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 3039, 3041, 4255, 4257, 8513, 70001, 136193])
def test_ray_counts_around_the_warps_share(ctx, n):
    """A launch of few rays spreads them over its warps: one ray a warp, the
    last warp short, two or more a warp, up to full warps (152 SMs x 7 or 5
    blocks x 4 warps), meshes and a two-level scene of both kinds."""
    from vermeer_gb300 import scenes
    v, ip = scenes.triangle_soup(1500, 11, edge=0.06)
    vm, im = scenes.motion_soup(700, 12, velocity=0.1, edge=0.06)
    gs, gm = ctx.mesh_build(v, ip), ctx.mesh_build(vm, im, keys=2, motion_mode=1)
    rays = _rays(n, 5)
    scene_rays = rays[np.isfinite(rays[:, :7]).all(1)] if n > 33 else scenes.incoherent_rays(n, 5)
    try:
        for shadow in (False, True):
            got = {}
            for k in (0, 45):
                ctx.set_tuning(kernel=k)
                r = [ctx.trace_mesh(g, rays, shadow=shadow) for g in (gs, gm)]
                for geoms in ([gs], [gs, gm]):
                    ctx.scene_build(geoms)
                    r.append(ctx.trace_scene(scene_rays, shadow=shadow))
                got[k] = r
            for a, b in zip(got[0], got[45]):
                for o in OUT:
                    x, y = (z[o].view(np.uint32) if z[o].dtype == np.float32 else z[o] for z in (a, b))
                    assert np.array_equal(x, y), (o, shadow)
    finally:
        ctx.set_tuning()


@pytest.mark.parametrize("kind", ["clean", "swapped", "nan", "inf"])
@pytest.mark.parametrize("moving", [False, True])
def test_top_level_copies_equal_the_nodes(ctx, kind, moving):
    """A top level over meshes, a sphere and (moving) motion and transformed
    meshes, its boxes as an upload may hold them."""
    from vermeer_gb300 import scenes
    rng = np.random.default_rng(9)
    geoms = []
    for k in range(9):
        v, ip = scenes.triangle_soup(200 + 90 * k, 50 + k, lo=0.1 * k, hi=0.1 * k + 0.4, edge=0.05)
        if moving and k % 3 == 1:
            v = np.concatenate([v, v + np.float32(0.05) * rng.standard_normal(3).astype(np.float32)])
            geoms.append(ctx.mesh_build(v, ip, keys=2, motion_mode=1))
        else:
            geoms.append(ctx.mesh_build(v, ip))
            if moving and k % 3 == 2:
                ctx.mesh_set_transform(geoms[-1], [1, 0.1, 0, 0, -0.1, 1, 0, 0, 0, 0, 0.9, 0, 0.05, 0, 0.1, 1])
    geoms.append(ctx.sphere_add((0.4, 0.5, 0.6), 0.15))
    ctx.scene_build(geoms)
    if kind != "clean":
        e = ctx.scene_export(len(geoms))
        if e["keys"] == 1:
            nodes, boxes = e["nodes"].copy(), np.ascontiguousarray(e["nodes"]["boxes"])
            _spoil(boxes, kind)
            nodes["boxes"] = boxes
            ctx.scene_upload(e["geom_order"], nodes=nodes)
        else:
            boxes = e["mboxes"].copy()
            _spoil(boxes, kind)
            ctx.scene_upload(e["geom_order"], mnodes=e["mnodes"], mboxes=boxes, keys=e["keys"])
    rays = _rays(4099, 13)
    try:
        for shadow in (False, True):
            got = {}
            for k in (0, 13, 45):
                ctx.set_tuning(kernel=k)
                got[k] = ctx.trace_scene(rays, shadow=shadow)
            for k in (13, 45):
                for o in OUT + ("geom",):
                    x, y = (z[o].view(np.uint32) if z[o].dtype == np.float32 else z[o] for z in (got[k], got[0]))
                    assert np.array_equal(x, y), (o, k, shadow)
    finally:
        ctx.set_tuning()


@pytest.mark.parametrize("keys", [1, 2, 3])
@pytest.mark.parametrize("tris", [40, 3000])
def test_rays_at_box_corners_equal_the_nodes(ctx, keys, tris):
    """Rays aimed at the vertices of axis-aligned right triangles, whose
    vertices are their boxes' corners: whether such a ray meets the box, and
    which triangle it hits, is decided by the last bit of every slab and edge
    product (and, with motion, of every lerp)."""
    from vermeer_gb300 import scenes
    rng = np.random.default_rng(17)
    c = rng.random((tris, 1, 3))
    off = rng.choice([-1.0, 1.0], (tris, 3)) * rng.uniform(0.02, 0.12, (tris, 3))
    ax = rng.integers(0, 3, tris)
    v = np.repeat(c, 3, 1)
    k = np.arange(tris)
    v[k, 1, ax] += off[k, ax]
    v[k, 2, (ax + 1) % 3] += off[k, (ax + 1) % 3]
    v = [(v + 0.3 * q * rng.standard_normal((tris, 1, 3))).astype(np.float32) for q in range(keys)]
    g = ctx.mesh_build(np.concatenate([x.reshape(-1, 3) for x in v]), np.arange(3 * tris, dtype=np.uint32), keys=keys,
                       motion_mode=1)
    n = 200_000
    time = rng.random(n).astype(np.float32)
    t = time * np.float32(keys - 1)
    k0 = np.floor(t).astype(int)
    f = (t - k0).astype(np.float32)[:, None]
    tri, vert = rng.integers(0, tris, n), rng.integers(0, 3, n)
    V = np.stack(v)
    p = (np.float32(1) - f) * V[k0, tri, vert] + f * V[np.minimum(k0 + 1, keys - 1), tri, vert]
    o = (p + rng.standard_normal((n, 3)).astype(np.float32)).astype(np.float32)
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3], rays[:, 3:6], rays[:, 6], rays[:, 7] = o, p - o, np.inf, time
    try:
        for shadow in (False, True):
            got = {}
            for k in (0, 13, 45):
                ctx.set_tuning(kernel=k)
                got[k] = ctx.trace_mesh(g, rays, shadow=shadow)
            for k in (13, 45):
                for q in OUT:
                    x, y = (z[q].view(np.uint32) if z[q].dtype == np.float32 else z[q] for z in (got[k], got[0]))
                    bad = np.nonzero(x != y)[0]
                    assert bad.size == 0, (q, k, shadow, bad.size, bad[:4])
    finally:
        ctx.set_tuning()
