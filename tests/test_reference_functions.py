"""The reference mode's functions in float32 pairs (df32.cuh) against the
float64 functions rounded to float32: every float32 input each takes, bit for
bit, and 2^27 pairs of sequence fractions for the sampling maps."""
import os
import shutil
import subprocess

import pytest

from vermeer_gb300 import build as vbuild

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_float32_pairs_round_as_float64(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "df32_check")
    r = subprocess.run([nvcc] + vbuild.NVCC_FLAGS + ["-I" + vbuild.CSRC, os.path.join(HERE, "df32_check.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 17
    bad = [row for row in rows if row[2] != "0"]
    assert not bad, r.stdout
