"""Rays whose time a motion mesh has no keys for, or is not a number, and boxes
that are not finite at a key.

A mesh is a miss for such a ray and the rest of the scene is not: the
while-while kernels against the step-scheduled mesh kernel and the single-loop
scene kernel (tuning kernel 0), bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OUT = ("prim", "t", "u", "v", "w")
OUTSIDE = (-0.25, -1e-30, np.nextafter(np.float32(1), np.float32(2)), 1.5, 7.0, np.inf, -np.inf)


def _rays(n, seed, times):
    """Times inside the keys, and each of times at every third ray in turn."""
    from vermeer_gb300 import scenes
    r = scenes.incoherent_rays(n, seed)
    r[:, 7] = scenes.uniform(seed, n, 77).astype(np.float32)
    at = np.arange(0, n, 3)
    r[at, 7] = np.asarray(times, np.float32)[(at // 3) % len(times)]
    return r


def _equal_to_kernel_0(ctx, trace, outputs):
    got = {}
    try:
        for shadow in (False, True):
            for k in (0, 13, 45):
                ctx.set_tuning(kernel=k)
                got[shadow, k] = trace(shadow)
            for k in (13, 45):
                for o in outputs:
                    x, y = (z[o].view(np.uint32) if z[o].dtype == np.float32 else z[o]
                            for z in (got[shadow, k], got[shadow, 0]))
                    bad = np.nonzero(x != y)[0]
                    assert bad.size == 0, (o, k, shadow, bad.size, bad[:4])
    finally:
        ctx.set_tuning()
    return got[False, 45]


def _static_top_over_moving_meshes(ctx, n_geoms, tris, keys):
    """A static top level uploaded over meshes of which two in three move (of
    those one in two has a transform as well) and a sphere: the top level of the
    meshes as they are at the first key."""
    from vermeer_gb300 import scenes
    still, geoms = [], []
    rng = np.random.default_rng(23)
    for k in range(n_geoms):
        v, ip = scenes.triangle_soup(tris + 40 * k, 80 + k, lo=0.1 * (k % 7), hi=0.1 * (k % 7) + 0.4, edge=0.06)
        still.append(ctx.mesh_build(v, ip))
        if k % 3 == 0:
            geoms.append(still[-1])
            continue
        step = np.float32(0.02) * rng.standard_normal(3).astype(np.float32)
        geoms.append(ctx.mesh_build(np.concatenate([v + np.float32(q) * step for q in range(keys)]), ip, keys=keys,
                                    motion_mode=1))
        if k % 3 == 2:
            ctx.mesh_set_transform(geoms[-1], [1, 0.02, 0, 0, -0.02, 1, 0, 0, 0, 0, 1, 0, 0.01, 0, 0.02, 1])
    still.append(ctx.sphere_add((0.4, 0.5, 0.6), 0.15))
    geoms.append(still[-1])
    ctx.scene_build(still)
    e = ctx.scene_export(len(still))
    assert e["keys"] == 1
    moved = dict(zip(still, geoms))
    ctx.scene_upload(np.array([moved[g] for g in e["geom_order"]], np.uint32), nodes=e["nodes"])
    return geoms


@pytest.mark.parametrize("n_geoms,tris", [(2, 20), (9, 200), (40, 60)])
@pytest.mark.parametrize("keys", [2, 3])
def test_static_top_level_over_moving_meshes(ctx, n_geoms, tris, keys):
    geoms = _static_top_over_moving_meshes(ctx, n_geoms, tris, keys)
    rays = _rays(8191, 41, OUTSIDE)
    r = _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_scene(rays, shadow=shadow), OUT + ("geom",))
    still = np.isin(r["geom"], [g for k, g in enumerate(geoms) if k % 3 == 0 or k == n_geoms] + [-1])
    assert still[::3].all() and not still.all()


@pytest.mark.parametrize("n_geoms,tris", [(2, 20), (9, 200)])
def test_nan_time_under_a_static_top_level(ctx, n_geoms, tris):
    geoms = _static_top_over_moving_meshes(ctx, n_geoms, tris, 2)
    rays = _rays(4099, 43, (np.nan,))
    r = _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_scene(rays, shadow=shadow), OUT + ("geom",))
    still = np.isin(r["geom"], [g for k, g in enumerate(geoms) if k % 3 == 0 or k == n_geoms] + [-1])
    assert still[::3].all() and not still.all()


@pytest.mark.parametrize("keys", [2, 3])
@pytest.mark.parametrize("tris", [1, 17, 1500])
def test_times_without_keys_miss_a_motion_mesh(ctx, keys, tris):
    from vermeer_gb300 import scenes
    v, ip = scenes.triangle_soup(tris, 11, edge=0.2 if tris < 100 else 0.06)
    step = np.float32(0.05) * scenes.unit_sphere(5, v.shape[0], 3).astype(np.float32)
    g = ctx.mesh_build(np.concatenate([v + np.float32(q) * step for q in range(keys)]), ip, keys=keys, motion_mode=1)
    rays = _rays(4099, 47, OUTSIDE + (np.nan,))
    r = _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_mesh(g, rays, shadow=shadow), OUT)
    assert (r["prim"][::3] == -1).all() and ((r["prim"] >= 0).any() or tris == 1)
    stats = []
    try:
        for k in (0, 13, 45):
            ctx.set_tuning(kernel=k)
            c = ctx.trace_mesh(g, rays, counters=True)["stats"]
            stats.append([c[q] for q in ("node_visits", "leaf_visits", "tri_tests")])
    finally:
        ctx.set_tuning()
    assert stats[1] == stats[0] and stats[2] == stats[0], stats
    # the same mesh under a top level that moves with it, and one that is still
    # beside it: nothing of such a scene is met
    w, iw = scenes.triangle_soup(40, 12, edge=0.2)
    ctx.scene_build([g, ctx.mesh_build(w, iw)])
    r = _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_scene(rays, shadow=shadow), OUT + ("geom",))
    assert (r["geom"][::3] == -1).all() and ((r["geom"] >= 0).any() or tris == 1)


def _reach_to_infinity(boxes, kind):
    """Planes at infinity, on one side or both, along one axis or all, in every
    third node (boxes: [keys, nodes, 24], min planes of the four children by axis,
    then max planes)."""
    b = boxes[:, ::3]
    axes = range(3) if kind.startswith("all") else (1,)
    for a in axes:
        if kind.endswith("below") or kind.endswith("both"):
            b[..., 4 * a:4 * a + 4] = -np.inf
        if kind.endswith("above") or kind.endswith("both"):
            b[..., 12 + 4 * a:16 + 4 * a] = np.inf
    return boxes


@pytest.mark.parametrize("kind", ["one_below", "one_above", "one_both", "all_below", "all_above", "all_both"])
@pytest.mark.parametrize("keys", [2, 3])
@pytest.mark.parametrize("tris", [3, 17, 1500])
def test_motion_boxes_at_infinity(ctx, kind, keys, tris):
    """At a key such a plane lerps to 0 * inf, a NaN: the slab test must take
    the box's other plane for it, as the node walk does."""
    from vermeer_gb300 import scenes
    v, ip = scenes.triangle_soup(tris, 11, edge=0.2 if tris < 100 else 0.06)
    step = np.float32(0.05) * scenes.unit_sphere(5, v.shape[0], 3).astype(np.float32)
    v = np.concatenate([v + np.float32(q) * step for q in range(keys)])
    e = ctx.mesh_export(ctx.mesh_build(v, ip, keys=keys, motion_mode=1))
    boxes = _reach_to_infinity(e["mboxes"].copy().reshape(keys, -1, 24), kind)
    g = ctx.mesh_upload(v, e["idxp"], e["accel_idx"], mnodes=e["mnodes"], mboxes=boxes, bounds=e["bounds"], keys=keys,
                        motion_mode=1)
    rays = _rays(4099, 53, (0.0, 1.0, 0.5, 0.25))
    _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_mesh(g, rays, shadow=shadow), OUT)
    w, iw = scenes.triangle_soup(40, 12, edge=0.2)
    ctx.scene_build([g, ctx.mesh_build(w, iw)])
    t = ctx.scene_export(2)
    assert t["keys"] == keys
    ctx.scene_upload(t["geom_order"], mnodes=t["mnodes"],
                     mboxes=_reach_to_infinity(t["mboxes"].copy().reshape(keys, -1, 24), kind), keys=keys)
    _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_scene(rays, shadow=shadow), OUT + ("geom",))


@pytest.mark.parametrize("keys,tris,nodes", [(1, 780, 32), (1, 800, 33), (2, 303, 16), (2, 305, 17), (3, 241, 10),
                                             (3, 237, 11)])
@pytest.mark.parametrize("spoil", [False, True])
def test_trees_around_the_size_whose_copies_the_host_makes(ctx, keys, tris, nodes, spoil):
    """Up to 32 nodes times keys, and just above; spoil: a NaN plane in the last
    node."""
    from vermeer_gb300 import scenes
    v, ip = scenes.triangle_soup(tris, 11, edge=0.06)
    step = np.float32(0.05) * scenes.unit_sphere(5, v.shape[0], 3).astype(np.float32)
    v = np.concatenate([v + np.float32(q) * step for q in range(keys)])
    g = ctx.mesh_build(v, ip, keys=keys, motion_mode=1)
    e = ctx.mesh_export(g)
    assert len(e["nodes" if keys == 1 else "mnodes"]) == nodes
    if spoil and keys == 1:
        n = e["nodes"].copy()
        n["boxes"].reshape(-1, 24)[-1, 13] = np.nan
        g = ctx.mesh_upload(v, e["idxp"], e["accel_idx"], nodes=n, bounds=e["bounds"])
    elif spoil:
        b = e["mboxes"].copy().reshape(keys, -1, 24)
        b[-1, -1, 13] = np.nan
        g = ctx.mesh_upload(v, e["idxp"], e["accel_idx"], mnodes=e["mnodes"], mboxes=b, bounds=e["bounds"], keys=keys,
                            motion_mode=1)
    rays = _rays(4099, 59, (0.0, 1.0, 0.5))
    r = _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_mesh(g, rays, shadow=shadow), OUT)
    assert (r["prim"] >= 0).any()


@pytest.mark.parametrize("n_geoms", [1, 2, 60, 80])
@pytest.mark.parametrize("moving", [False, True])
def test_top_levels_around_the_size_whose_copies_the_host_makes(ctx, n_geoms, moving):
    from vermeer_gb300 import scenes
    geoms = []
    for k in range(n_geoms):
        v, ip = scenes.triangle_soup(30, 200 + k, lo=0.01 * (k % 60), hi=0.01 * (k % 60) + 0.4, edge=0.08)
        if moving and k % 4 == 0:
            geoms.append(ctx.mesh_build(np.concatenate([v, v + np.float32(0.02)]), ip, keys=2, motion_mode=1))
        else:
            geoms.append(ctx.mesh_build(v, ip))
    ctx.scene_build(geoms)
    rays = _rays(4099, 61, (0.0, 1.0, 0.5))
    r = _equal_to_kernel_0(ctx, lambda shadow: ctx.trace_scene(rays, shadow=shadow), OUT + ("geom",))
    assert (r["geom"] >= 0).any()
