"""The parallel merge of a chunk's runs where it can go wrong: spans of one
sample up to the whole ray (one piece, a few, more pieces than a chunk has
lanes), more candidate runs per column than a lane records, columns whose
spans overlap and hide one another, and cells whose clip-top test depends on
the horizon (an eye above the scene's top).  Every lane count against the
oracle: ray-buffer words, depths and hit records bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import Frame, assert_rays_equal

pytestmark = pytest.mark.gpu

N, SY = 64, 256


def _volume(kind: str) -> np.ndarray:
    """Solid voxels [z][y][x], y from the top."""
    rng = np.random.default_rng(11)
    v = np.zeros((N, SY, N), bool)
    z, y, x = np.ogrid[:N, :SY, :N]
    v[:, SY - 4:, :] = True
    if kind == "walls":  # tall faces one step from the eye: spans of the whole ray
        v |= (((x % 16) == 0) | ((z % 16) == 0)) & (y > 20)
        v[28:37, :240, 28:37] = False
    elif kind == "slats":  # up to 16 thin runs per column, hiding one another
        v |= ((y // 8) % 2 == 0) & (y > 100) & (((x // 4) + (z // 4)) % 2 == 0)
        v |= ((y // 4) % 2 == 0) & (y > 100) & (((x // 4) + (z // 4)) % 2 == 1)
        v[26:39, :, 26:39] = False
    else:  # single voxels scattered through the air
        v |= rng.random((N, SY, N)) < 0.02
        v[26:39, 90:170, 26:39] = False
    return v


@pytest.fixture(scope="module", params=["walls", "slats", "dust"])
def scene(request, rle, po, torch_cuda):
    v = _volume(request.param)
    levels = []
    bits, sy = po.pack_bits(v), SY
    n = N
    for m in range(3):
        _, words = po.encode_mip(bits, n, sy, n, m)
        levels.append((n, sy, n, words))
        bits = po.mipmap(bits, n, sy, n)
        n, sy = n // 2, sy // 2
    data = po.write_rle4(levels)
    yield request.param, rle.Scene.from_bytes(data), po.OracleScene.from_rle4(data)
    rle.tuning_set(0, 0, 0, 0)


@pytest.mark.parametrize("lanes", [8, 16, 32])
@pytest.mark.parametrize("samples", [24, 512, 4096])
def test_merge_bit_exact(rle, po, torch_cuda, scene, lanes, samples):
    kind, s, o = scene
    rle.tuning_set(lanes, 0, 0, 0)
    try:
        # inside the clearing, looking ahead and steeply down; above the top
        for height, yaw, pitch in ((130.0, 20.0, -8.0), (120.0, 135.0, 70.0), (SY + 30.0, 250.0, -35.0)):
            cam = rle.camera(32.4, 32.6, height, yaw, pitch, scene_height=SY)
            rm = rle.raymap_build(cam, rle.view_params(96, 64, samples=samples, mip_distance=40, z_far=400))
            gpu = Frame(torch_cuda, rle, s, rm, counters=False).rays_host()
            orc = po.render_rays(po.raymap_from_product(rm), o, want_hits=True)
            assert_rays_equal(gpu, orc, f"{kind} lanes {lanes} samples {samples} height {height} pitch {pitch}")
    finally:
        rle.tuning_set(0, 0, 0, 0)
