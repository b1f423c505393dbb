"""What a tuning may cost against the default one: tunings change how rays are
scheduled, and a kernel that loses its warps' convergence shows here first."""
import time

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
