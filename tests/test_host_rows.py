"""Host callers' rows laid out by the device: rays of 8 floats against the same
rays passed as arrays, at the ends of warps, blocks, the reordering threshold
and the staging chunk; the guide's n x 3 inputs at ragged tile sizes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 31, 257, 65537, (1 << 20) + 3])
def test_ray_rows_equal_arrays(ctx, n):
    from vermeer_gb300 import _lib, scenes
    v, ip = scenes.triangle_soup(1500, 51, edge=0.05)
    vm, im = scenes.motion_soup(500, 52, velocity=0.1, edge=0.05)
    geoms = [ctx.mesh_build(v, ip), ctx.mesh_build(vm, im, keys=2, motion_mode=1)]
    ctx.scene_build(geoms)
    rays = scenes.incoherent_rays(max(n, 1), 53)[:n]
    rays[:, 7] = scenes.uniform(54, max(n, 1), 1).astype(np.float32).ravel()[:n]
    cols = np.ascontiguousarray(rays.T)
    ptr = [ctypes.c_void_p(cols.ctypes.data + 4 * n * k) for k in range(8)]
    for geom in (*geoms, None):
        rows = ctx.trace_scene(rays) if geom is None else ctx.trace_mesh(geom, rays)
        names = [k for k in ("prim", "geom", "t", "u", "v", "w") if k in rows]
        arr = {k: np.empty(n, rows[k].dtype) for k in names}
        h = _lib.Hits(*[arr[k].ctypes.data_as(ctypes.c_void_p) if k in arr else None
                        for k in ("prim", "geom", "t", "u", "v", "w")])
        call = (ctypes.byref(_lib.Rays(*ptr)), n, 0, ctypes.byref(h), None)
        rc = ctx.L.vmr_trace_scene(ctx.h, *call) if geom is None else ctx.L.vmr_trace_mesh(ctx.h, geom, *call)
        assert rc == 0
        for k in names:
            assert np.array_equal(rows[k].view(np.uint32), arr[k].view(np.uint32)), (geom, k)


def test_ray_rows_refusals(ctx):
    from vermeer_gb300 import _lib, scenes
    g = ctx.mesh_build(*scenes.triangle_soup(50, 55, edge=0.2))
    rays = scenes.incoherent_rays(8, 56)
    p, h = rays.ctypes.data_as(ctypes.c_void_p), ctypes.byref(_lib.Hits())
    assert ctx.L.vmr_trace_mesh_rows(ctx.h, g, p, 8, 2, h, None) == -1  # device rays
    assert ctx.L.vmr_trace_mesh_rows(ctx.h, g, None, 8, 0, h, None) == -1
    assert ctx.L.vmr_trace_mesh_rows(ctx.h, 0xffffffff, p, 8, 0, h, None) == -1


@pytest.mark.parametrize("n", [1, 127, 129, 1025])
def test_guide_rows_are_read_in_place(ctx, n):
    rng = np.random.default_rng(57)
    pos, nrm, wo = (rng.standard_normal((1100, 3)).astype(np.float32) for _ in range(3))
    lo, hi = np.full(3, -4, np.float32), np.full(3, 4, np.float32)
    ctx.guide_init(1)
    want = ctx.guide_forward(pos, nrm, wo, lo, hi)
    got = ctx.guide_forward(pos[:n], nrm[:n], wo[:n], lo, hi)
    assert np.array_equal(got.view(np.uint32), want[:n].view(np.uint32))  # rows are independent
