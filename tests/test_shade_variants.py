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


@pytest.mark.parametrize("w", [1, 31, 32, 33, 255, 257])
@pytest.mark.parametrize("kind", ["room", "furnace"])
def test_queue_remainders(ctx, kind, w):
    """The hits that wait for a full group: the iterations in one batch, whose
    rounds leave other remainders than batches of one iteration each."""
    from vermeer_gb300 import scenes
    ctx.load_scene(scenes.small_room_ext(300, seed=4) if kind == "room" else scenes.furnace(subdiv=4))
    a, _ = ctx.render_path(w, 1, 0, 37, 9, max_depth=5)
    b, _ = ctx.render_path(w, 1, 0, 37, 9, max_depth=5, max_batch_samples=w)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
