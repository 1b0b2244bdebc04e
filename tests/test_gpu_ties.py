"""Column rays whose DDA axes meet at equal distances -- an eye at a multiple of
1/16 of a cell looking straight down or along a diagonal -- over ground where
every column has a height and a colour of its own, so that a ray that steps
along the wrong axis at a tie draws other words: ray-buffer words, depths and
hit records against the oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import Frame, assert_rays_equal

pytestmark = pytest.mark.gpu

N, SY = 64, 256
# eye x, z, yaw, pitch; screen width, height; samples per ray; first level distance
POSES = [
    (34.5, 36.5, 270, -90, 128, 96, 128, 64),
    (47.5, 60.5, 90, -90, 128, 96, 128, 64),
    (31.5, 1.5, 90, -90, 128, 96, 128, 64),
    (58.5, 46.5, 225, -90, 64, 64, 128, 256),
    (49.5, 54.5, 45, -90, 64, 64, 64, 256),
    (109.0, 563.0, 180, -45, 64, 64, 64, 256),
    (534.75, 677.25, 90, -45, 160, 120, 64, 40),
]


def rough_ground(po) -> bytes:
    """.rle4 bytes of one level: a column of random height on every cell."""
    rng = np.random.default_rng(5)
    top = rng.integers(SY - 90, SY - 4, (N, 1, N))
    v = np.arange(SY)[None, :, None] >= top
    colours = rng.integers(0, 1 << 16, (N, SY, N), dtype=np.uint16)
    _, words = po.encode_mip(po.pack_bits(v), N, SY, N, 0, colours.reshape(-1))
    return po.write_rle4([(N, SY, N, words)])


@pytest.mark.parametrize("pose", POSES, ids=lambda p: f"{p[0]}-{p[1]}-{p[2]}-{p[3]}")
def test_ties_bit_exact(rle, po, torch_cuda, pose):
    x, z, yaw, pitch, width, height, samples, level = pose
    data = rough_ground(po)
    cam = rle.camera(x, z, 130.0, yaw, pitch, scene_height=SY)
    rm = rle.raymap_build(cam, rle.view_params(width, height, samples=samples, mip_distance=level, z_far=400))
    with rle.Scene.from_bytes(data) as scene:
        gpu = Frame(torch_cuda, rle, scene, rm, counters=False).rays_host()
    orc = po.render_rays(po.raymap_from_product(rm), po.OracleScene.from_rle4(data), want_hits=True)
    assert_rays_equal(gpu, orc, str(pose))
