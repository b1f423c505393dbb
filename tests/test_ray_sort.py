"""The ray reordering at its edges: every key width (the scan's shares are
uneven at the smallest), batches just past the threshold, rays with times
against a static mesh (the record copy carries none), an odd number of paths
in a render's queue sort.  Against the unsorted kernels, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [3, 4, 5])
@pytest.mark.parametrize("n", [65536, 65537, 99991])
def test_sorted_traces_equal_unsorted(ctx, bits, n):
    from vermeer_gb300 import scenes
    import torch
    v, ip = scenes.triangle_soup(3000, 41, edge=0.05)
    vm, im = scenes.motion_soup(1500, 42, velocity=0.1, edge=0.05)
    geoms = [ctx.mesh_build(v, ip), ctx.mesh_build(vm, im, keys=2, motion_mode=1)]
    rays = scenes.incoherent_rays(n, 43)
    rays[:, 7] = scenes.uniform(44, n, 1).astype(np.float32)
    rays[::5, 0:3] = 0.25  # a crowded bucket
    dev = torch.from_numpy(np.ascontiguousarray(rays.T)).cuda()
    ctx.scene_build([geoms[0]])
    try:
        for shadow in (False, True):
            got = []
            for kernel in (45 & ~8, 45):
                ctx.set_tuning(kernel=kernel, sort_bits=bits)
                r = [ctx.trace_mesh(g, rays, shadow=shadow) for g in geoms]
                r += [ctx.trace_mesh(g, dev, shadow=shadow) for g in geoms]
                r.append(ctx.trace_scene(rays, shadow=shadow))
                ctx.sync()
                got.append(r)
            for a, b in zip(*got):
                for k in ("prim", "t", "u", "v", "w"):
                    x, y = (np.asarray(z[k].cpu() if hasattr(z[k], "cpu") else z[k]) for z in (a, b))
                    assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (k, shadow)
    finally:
        ctx.set_tuning()


def test_queue_sort_with_an_odd_number_of_paths(ctx):
    from vermeer_gb300 import scenes
    ctx.load_scene(scenes.small_room_ext(500, seed=3))
    a, _ = ctx.render_path(257, 257, 0, 1, 5, max_depth=3)
    b, _ = ctx.render_path(257, 257, 0, 1, 5, max_depth=3, sort_queues=True)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("n", [65536, 70001])
def test_sorted_scene_records_equal_unsorted(ctx, n):
    """Several meshes and a sphere, which reads the ray again: record copies
    against the rays in input order."""
    from vermeer_gb300 import scenes
    geoms = [ctx.mesh_build(*scenes.triangle_soup(800, 45 + k, edge=0.08)) for k in range(2)]
    geoms.append(ctx.sphere_add((0.5, 0.5, 0.5), 0.2))
    ctx.scene_build(geoms)
    rays = scenes.incoherent_rays(n, 48)
    rays[1::3, 6] = 0.4  # some with a finite reach
    try:
        for shadow in (False, True):
            got = []
            for kernel in (45 & ~8, 45, 45 & ~32):
                ctx.set_tuning(kernel=kernel)
                got.append(ctx.trace_scene(rays, shadow=shadow))
            assert (got[0]["geom"] == geoms[2]).any() and (got[0]["geom"] == geoms[0]).any()
            for g in got[1:]:
                for k in ("prim", "geom", "t", "u", "v", "w"):
                    assert np.array_equal(got[0][k].view(np.uint32), g[k].view(np.uint32)), (k, shadow)
    finally:
        ctx.set_tuning()
