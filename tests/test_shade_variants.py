"""The two forms of the path tracer's shading kernel (batches below and from
4,194,304 paths on): one image rendered in one large batch and in small ones,
bit for bit, over every lobe, light kind and Russian roulette, and over a
scene most rays miss."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["room", "furnace"])
def test_large_and_small_batches_shade_alike(ctx, kind):
    from vermeer_gb300 import scenes
    ctx.load_scene(scenes.small_room_ext(1500, seed=3) if kind == "room" else scenes.furnace(subdiv=6))
    w, h, it = 521, 509, 16  # 4,242,224 paths; an odd last block
    a, st = ctx.render_path(w, h, 0, it, 5, max_depth=6)
    assert st["samples"] == w * h * it
    b, _ = ctx.render_path(w, h, 0, it, 5, max_depth=6, max_batch_samples=w * h * 3)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
