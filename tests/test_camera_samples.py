"""Camera samples: the float32-pair expressions against float64's, and images at
the raster enumeration's largest widths, heights and a late iteration, against
the oracle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from vermeer_gb300 import build as vbuild, scenes

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_camera_expressions_round_as_float64(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "camera_check")
    r = subprocess.run([nvcc] + vbuild.NVCC_FLAGS + ["-I" + vbuild.CSRC, os.path.join(HERE, "camera_check.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 2 and all(row[2] == "0" for row in rows), r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,first", [(4096, 2, 0), (2, 4096, 0), (7, 5, 70000)])
def test_raster_edges_match_oracle(ctx, orc, w, h, first):
    """The tolerance and its reasons are test_render.py's."""
    room = scenes.small_room(512, seed=5)
    ctx.load_scene(room)
    got, _ = ctx.render(w, h, first, 1, 11)
    ref = orc.Render(room).run(w, h, first, 1, 11)
    ok = (np.abs(got - ref) <= 1e-5 * (1.0 + np.abs(ref))).all(-1)
    assert ok.mean() >= 0.999 and np.abs(got - ref).mean() <= 1e-6
