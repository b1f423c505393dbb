"""A scene changed between traces answers as one made that way at once."""
import numpy as np
import pytest

from conftest import assert_hits_equal

pytestmark = pytest.mark.gpu
OUT = ("prim", "geom", "t", "u", "v", "w")
XF = ([1, 0.1, 0, 0, -0.1, 1, 0, 0, 0, 0, 0.9, 0, 0.05, 0, 0.1, 1], [0.8, 0, 0, 0, 0, 1.1, 0, 0, 0, 0, 1, 0, 0, 0.1, 0, 1])


def _meshes(c, moving):
    from vermeer_gb300 import scenes
    geoms = []
    for k in range(5):
        v, ip = scenes.triangle_soup(150 + 40 * k, 60 + k, lo=0.1 * k, hi=0.1 * k + 0.5, edge=0.06)
        if moving and k % 2:
            geoms.append(c.mesh_build(np.concatenate([v, v + np.float32(0.03)]), ip, keys=2, motion_mode=1))
        else:
            geoms.append(c.mesh_build(v, ip))
    return geoms


@pytest.mark.parametrize("moving", [False, True])
def test_transforms_set_and_removed_between_traces(moving):
    import vermeer_gb300 as vg
    from vermeer_gb300 import scenes
    rays = scenes.incoherent_rays(3001, 9)
    rays[:, 7] = scenes.uniform(9, 3001, 7).astype(np.float32)

    def fresh(members, xf):
        c = vg.Context(0)
        geoms = _meshes(c, moving)
        for k, m in xf.items():
            c.mesh_set_transform(geoms[k], m)
        c.scene_build([geoms[k] for k in members])
        out = [c.trace_scene(rays, shadow=s) for s in (False, True)]
        c.close()
        return out

    c = vg.Context(0)
    geoms = _meshes(c, moving)
    members, xf = range(4), {}
    c.scene_build([geoms[k] for k in members])
    for step in ("as built", (1, XF[0]), (2, XF[1]), (1, XF[1]), (1, None), "rebuilt", (4, XF[0]), (2, None)):
        if step == "rebuilt":
            members = (4, 0, 2, 1)
            c.scene_build([geoms[k] for k in members])
        elif step != "as built":
            k, m = step
            c.mesh_set_transform(geoms[k], m)
            xf = {q: w for q, w in {**xf, k: m}.items() if w is not None}
        for shadow, ref in zip((False, True), fresh(members, xf)):
            assert_hits_equal(c.trace_scene(rays, shadow=shadow), ref, OUT, f"{step} {shadow}")
    c.close()
