"""A call that was refused leaves nothing behind that fails the next one: the
runtime keeps a failed call as the thread's last error, which launches are
checked with."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

W, H = 64, 48


def _refused(rle, what):
    if what == "batch memory":
        rle.Batch(1, 1 << 42, W)
    elif what == "batch device":
        rle.Batch(1, 1 << 16, W, device=63)
    elif what == "server memory":
        rle.Server(1 << 62, 1 << 42, max_samples=W)
    elif what == "server device":
        rle.Server(1 << 40, 1 << 16, max_samples=W, device=63)
    elif what == "scene device":
        rle.Scene.generate_on_device(rle.scenegen_default(64, 64, 64, 5), device=63)
    else:
        rle.bounds_check_read(63)


@pytest.mark.parametrize("what", ["batch memory", "batch device", "server memory", "server device", "scene device",
                                  "bounds device"])
def test_the_next_frame_is_drawn(rle, torch_cuda, what):
    torch = torch_cuda
    view = rle.view_params(W, H)
    n = rle.frame_workspace_bytes(view)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    colour = torch.empty(W * H, dtype=torch.int32, device="cuda")
    depth = torch.empty(W * H, dtype=torch.float32, device="cuda")
    cam = rle.camera(30.0, 21.0, 60.0, 20.0, -12.0, scene_height=64)
    with rle.Scene.from_bytes(rle.scenegen_rle4(rle.scenegen_default(64, 64, 64, 5))) as scene:
        with pytest.raises(rle.RLEError):
            _refused(rle, what)
        rle.render_frame(scene, cam, view, ws, n, colour, depth)
        torch.cuda.synchronize()
