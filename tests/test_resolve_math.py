"""The resolve's texture coordinates with only the terms that count against the
shader's arithmetic as it stands: the header the kernels include, compiled for
the host and compared over random cameras' uniforms and pixels, and its
division by a known divisor against IEEE division, bit for bit."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from gpu_util import assert_screen_equal, oracle_screen

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "rle-based-voxel-raycasting_gb300" / "csrc"


@pytest.mark.parametrize("seed", [1, 2])
def test_coordinates_equal_the_shader(seed, tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = tmp_path / "resolve_math_check"
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC),
           str(ROOT / "tests" / "c" / "resolve_math_check.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe), str(seed), "300"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    bad, bad_div, seen = map(int, r.stdout.split())
    assert (bad, bad_div) == (0, 0)
    assert seen > 1000000


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(8, 8), (33, 9), (32, 8), (31, 31), (257, 40), (640, 479)])
def test_resolve_tiles(rle, po, torch_cuda, size):
    """Screens around the tile's edges against the oracle's screen."""
    torch = torch_cuda
    w, h = size
    data = rle.scenegen_rle4(rle.scenegen_default(64, 64, 64, 5, caves=True))
    scene, oscene = rle.Scene.from_bytes(data), po.OracleScene.from_rle4(data)
    for yaw, pitch in ((20.0, -12.0), (200.0, 50.0)):
        cam = rle.camera(30.5, 21.25, 60.0, yaw, pitch, scene_height=64)
        view = rle.view_params(w, h, samples=64)
        n = rle.frame_workspace_bytes(view)
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        c = torch.empty(w * h, dtype=torch.int32, device="cuda")
        d = torch.empty(w * h, dtype=torch.float32, device="cuda")
        hit = torch.empty(w * h * 8, dtype=torch.uint8, device="cuda")
        rle.render_frame(scene, cam, view, ws, n, c, d, hit)
        torch.cuda.synchronize()
        got = c.cpu().numpy().view(np.uint32), d.cpu().numpy(), hit.cpu().numpy().view(rle.HIT_DTYPE)
        assert_screen_equal(got, oracle_screen(po, rle, oscene, cam, view), f"{size} yaw {yaw}")
    scene.free()
