"""The share of the device's memory the octant copies may take (octant_room)."""
import os
import subprocess

import pytest

from vermeer_gb300 import build as vbuild

GB = 10 ** 9


@pytest.mark.parametrize("held,more,total,room", [
    (0, 51 * 10 ** 6, 284 * GB, True),            # a million triangles
    (0, 365 * 10 ** 6, 284 * GB, True),           # the largest mesh
    (17 * GB, 365 * 10 ** 6, 284 * GB, True),
    (17 * GB, 750 * 10 ** 6, 284 * GB, True),     # to the sixteenth
    (17 * GB, 750 * 10 ** 6 + 1, 284 * GB, False),
    (0, 18 * GB, 284 * GB, False),
    (2 * GB, 1, 16 * GB, False),                  # a small device
    (0, GB, 16 * GB, True),
])
def test_copies_take_at_most_a_sixteenth(tmp_path, held, more, total, room):
    src, exe = str(tmp_path / "room.cpp"), str(tmp_path / "room")
    with open(src, "w") as f:
        f.write('#include <cstdio>\n#include "device.h"\nint main() {\n'
                f'  std::printf("%d", (int)vmr::octant_room({held}ull, {more}ull, {total}ull));\n}}\n')
    subprocess.run(["g++", "-std=c++17", "-I" + vbuild.CSRC, "-I" + vbuild.INCLUDE, src, "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout == str(int(room))


@pytest.mark.gpu
def test_copies_go_with_what_they_belong_to():
    """Meshes, top levels and flattened scenes made and replaced in one context
    leave no copies behind: the device's free memory comes back."""
    import numpy as np
    import torch
    import vermeer_gb300 as vg
    from vermeer_gb300 import scenes
    c = vg.Context(0)
    free = []
    v, ip = scenes.triangle_soup(3000, 3, edge=0.05)
    geoms = [c.mesh_build(v + np.float32(k), ip) for k in range(4)]
    vm, im = scenes.motion_soup(500, 12, velocity=0.1, edge=0.06)
    e = c.mesh_export(c.mesh_build(vm, im, keys=2, motion_mode=1))
    c.mesh_upload(vm, e["idxp"], e["accel_idx"], mnodes=e["mnodes"], mboxes=np.full_like(e["mboxes"], np.inf),
                  bounds=e["bounds"], keys=2, motion_mode=1)
    rays = scenes.incoherent_rays(5000, 3)
    first = None
    for k in range(12):
        c.scene_build(geoms[:2 + k % 3])
        r = c.trace_scene(rays)
        first = r if first is None else first
        if k % 3 == 0:
            assert np.array_equal(r["prim"], first["prim"]) and np.array_equal(r["t"], first["t"])
            free.append(torch.cuda.mem_get_info()[0])
    c.close()
    assert free[-1] == free[1]
