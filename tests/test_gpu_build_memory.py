"""Building a scene with little device memory left: the levels are encoded one
by one where the scratch of all of them does not fit, with the same result;
where that does not fit either, the build reports it and releases everything."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_little_memory(rle, torch_cuda):
    torch = torch_cuda
    p = rle.scenegen_default(1024, 256, 1024, 5, caves=True)
    p.nummaps = 4
    with rle.Scene.generate_on_device(p) as scene:
        nbytes = scene.info().device_bytes
        ref = [scene.copy_level(m) for m in range(4)]
    torch.cuda.empty_cache()
    # bytes per column: 32 of voxel bits, 46 of scratch; a quarter and less of it at the further levels
    n = 1024 * 1024
    block, extra = n * (32 * 4 // 3 + 46), n * 30 // 4
    built = refused = 0
    for spare in range(-extra - 16 * MB, extra + 32 * MB, 4 * MB):  # around block + scene, by less than the extra scratch
        free, _ = torch.cuda.mem_get_info()
        ballast = torch.empty(max(free - (block + nbytes + spare), 0), dtype=torch.uint8, device="cuda")
        try:
            with rle.Scene.generate_on_device(p) as scene:
                assert scene.info().device_bytes == nbytes
                for m in range(4):
                    for a, b in zip(ref[m], scene.copy_level(m)):
                        assert np.array_equal(a, b), (spare, m)
            built += 1
        except rle.RLEError as e:
            assert "cudaMalloc" in str(e), str(e)
            refused += 1
        del ballast
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] >= free - 4 * MB  # nothing kept
    assert built and refused
