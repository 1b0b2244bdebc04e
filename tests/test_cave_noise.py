"""The conversion-free cave noise against the generator's own, bit for bit: the
header the kernel includes, compiled for the host; and on the device grids at
either side of the coordinate limit against the host generator."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "rle-based-voxel-raycasting_gb300" / "csrc"


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_noise_equals_the_generators(seed, tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = tmp_path / "cave_noise_check"
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC),
           str(ROOT / "tests" / "c" / "cave_noise_check.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe), str(seed), "1000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    bad, bad_cave, points = map(int, r.stdout.split())
    assert (bad, bad_cave) == (0, 0)
    assert points == 1000000


@pytest.mark.gpu
@pytest.mark.parametrize("period", [0.001, 0.0025, 0.004, 1.0, 7.5, 400.0])
@pytest.mark.parametrize("size", [(8, 64, 8), (8, 128, 32), (64, 192, 8)])
def test_cave_periods(rle, torch_cuda, size, period):
    """Smallest grids and periods around the limit (0.001 .. 0.004)."""
    sx, sy, sz = size
    p = rle.scenegen_default(sx, sy, sz, 11, caves=True)
    p.nummaps = 1
    p.base_period = 8
    p.cave_period, p.cave_threshold, p.cave_y0, p.cave_y1 = period, 0.1, 1.0, float(sy)
    host, dev = rle.Scene.from_bytes(rle.scenegen_rle4(p)), rle.Scene.generate_on_device(p)
    for a, b in zip(host.copy_level(0), dev.copy_level(0)):
        assert np.array_equal(a, b)
    host.free()
    dev.free()
