"""What a tuning may cost against the default one: tunings change how rays are
scheduled, and a kernel that loses its warps' convergence shows here first."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_level_render_with_leaves_scanned_by_their_lanes(ctx):
    """Kernel 13 against 45 (the cooperative leaf scan).  1.3 to 1.4 times the
    default's time where the lanes of a warp scan their leaves together, above 4
    where they come to them one by one; fastest of nine renders of 2 to 4 ms."""
    from vermeer_gb300 import scenes
    ctx.load_scene(scenes.small_room(4096, seed=1))
    best = {}
    try:
        for k in (45, 13):
            ctx.set_tuning(kernel=k)
            t = []
            for _ in range(10):
                t0 = time.perf_counter()
                ctx.render_path(256, 256, 0, 4, 3, max_depth=5, two_level=True)
                t.append(time.perf_counter() - t0)
            best[k] = min(t[1:])
    finally:
        ctx.set_tuning()
    assert best[13] < 2.2 * best[45], best


def test_blocks_of_256_threads_stay_resident(ctx):
    """Kernel 1 at 256 threads a block against kernel 5 (128 threads, capped
    registers): 1.03 times its time where three such blocks fit an SM, 1.25 where two
    do; fastest of eleven traces of about 2 ms, device rays."""
    import torch
    from vermeer_gb300 import scenes
    v, ip = scenes.triangle_soup(200003, 2, edge=0.0085)
    g = ctx.mesh_build(v, ip)
    rays = torch.from_numpy(np.ascontiguousarray(scenes.incoherent_rays(1 << 20, 1).T)).cuda()
    torch.cuda.synchronize()
    best = {}
    try:
        for kernel, block in ((5, 0), (1, 256)):
            ctx.set_tuning(kernel=kernel, block=block)
            t = []
            for _ in range(12):
                t0 = time.perf_counter()
                ctx.trace_mesh(g, rays)
                ctx.sync()
                t.append(time.perf_counter() - t0)
            best[kernel] = min(t[1:])
    finally:
        ctx.set_tuning()
    assert best[1] < 1.15 * best[5], best
