"""The device encoder takes tensors that the current torch stream is still
computing: what it encodes is what that stream leaves in them."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_encode import _levels

pytestmark = pytest.mark.gpu

N, SY = 256, 128


@pytest.mark.parametrize("side", [False, True])
def test_encoder_waits_for_the_current_stream(rle, torch_cuda, side):
    torch = torch_cuda
    rng = np.random.default_rng(3)
    bits = torch.from_numpy(rng.integers(0, 256, N * N * SY // 8, dtype=np.uint8)).cuda()
    colours = torch.from_numpy(rng.integers(-32768, 32767, N * N * SY, dtype=np.int16)).cuda()
    late_bits, late_colours = torch.zeros_like(bits), torch.zeros_like(colours)
    a = torch.randn(8192, 8192, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        for _ in range(8):  # tens of milliseconds
            b = a @ a
        late_bits.copy_(bits)
        late_colours.copy_(colours)
        with rle.Scene.encode_on_device(late_bits, late_colours, N, SY, N, 3) as scene:
            _, got = _levels(rle, scene)
    torch.cuda.synchronize()
    del a, b
    with rle.Scene.encode_on_device(bits, colours, N, SY, N, 3) as scene:
        _, want = _levels(rle, scene)
    for m, (w, g) in enumerate(zip(want, got)):
        assert np.array_equal(w[3], g[3]) and np.array_equal(w[4], g[4]), f"level {m}"


def test_encoder_while_a_stream_is_captured(rle, torch_cuda):
    """The current stream being captured has run nothing: the build does not
    wait for it and does not join the capture."""
    torch = torch_cuda
    rng = np.random.default_rng(4)
    bits = torch.from_numpy(rng.integers(0, 256, 64 * 64 * 64 // 8, dtype=np.uint8)).cuda()
    x = torch.zeros(1024, device="cuda")
    with rle.Scene.encode_on_device(bits, None, 64, 64, 64, 2) as scene:
        _, want = _levels(rle, scene)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        x += 1
        scene = rle.Scene.encode_on_device(bits, None, 64, 64, 64, 2)
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.min()) == float(x.max()) == 2.0
    _, got = _levels(rle, scene)
    scene.free()
    for w, g in zip(want, got):
        assert np.array_equal(w[3], g[3]) and np.array_equal(w[4], g[4])


@pytest.mark.parametrize("device", [-1, 99])
def test_encoder_refuses_a_device_that_is_not_there(rle, torch_cuda, device):
    bits = torch_cuda.zeros(64 * 64 * 64 // 8, dtype=torch_cuda.uint8, device="cuda")
    with pytest.raises(rle.RLEError) as e:
        rle.Scene.encode_on_device(bits, None, 64, 64, 64, 2, device=device)
    assert e.value.name == "RLE_ERR_INVALID_ARG"
