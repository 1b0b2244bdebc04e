"""The device encoder where its kernels change course, against the oracle: rows
shorter than a warp, heights around the 64-voxel words, runs that cross and end
at words, and columns so full of runs that a warp's words go through the stage
in many turns."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_encode import _levels, _oracle_levels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["alternating", "noise", "solid", "words", "empty"])
@pytest.mark.parametrize("dims", [(8, 1024, 8), (16, 65, 8), (8, 64, 32), (64, 127, 16), (32, 129, 32)])
@pytest.mark.parametrize("with_colours", [False, True])
def test_edges(rle, po, torch_cuda, dims, kind, with_colours):
    torch = torch_cuda
    sx, sy, sz = dims
    rng = np.random.default_rng(sx + sy)
    j = np.arange(sy)[None, :, None]
    vol = {"alternating": (j + np.arange(sx)[None, None, :]) % 2 == 0,
           "noise": rng.random((sz, sy, sx)) < 0.5,
           "solid": j >= 0,
           "words": (j // 64) % 2 == 1,
           "empty": j < 0}[kind]
    vol = np.ascontiguousarray(np.broadcast_to(vol, (sz, sy, sx)))
    bits = po.pack_bits(vol)
    colours = rng.integers(0, 65536, sx * sy * sz, dtype=np.uint16) if with_colours else None
    levels = min(sx, sz).bit_length() - 3  # the oracle's mips are whole bytes of 8 voxels
    want = _oracle_levels(po, bits, colours, sx, sy, sz, levels)
    d_col = torch.from_numpy(colours.view(np.int16)).cuda() if with_colours else None
    with rle.Scene.encode_on_device(torch.from_numpy(bits).cuda(), d_col, sx, sy, sz, levels) as scene:
        _, got = _levels(rle, scene)
    for m, (a, b) in enumerate(zip(want, got)):
        assert a[:3] == b[:3], f"level {m} size"
        assert np.array_equal(a[4], b[4]), f"level {m} slab words"
        assert np.array_equal(a[3], b[3]), f"level {m} table"
