"""A request whose rays would never end is refused where it is made, so that it
takes no other request of its launch with it: at the server's submit, and by
frames and batches before anything is launched (the rule itself is compared
with the march's loop on the host in test_march_ends.py)."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

W, H = 64, 48


def test_refused_at_submit_others_served(rle, torch_cuda):
    torch = torch_cuda
    cam = rle.camera(30.0, 21.0, 60.0, 20.0, -12.0, scene_height=64)
    good, endless = rle.view_params(W, H, mip_distance=16), rle.view_params(W, H, mip_distance=1)
    outs = [(torch.empty(W * H, dtype=torch.int32, device="cuda"), torch.empty(W * H, device="cuda")) for _ in range(4)]
    with rle.Scene.from_bytes(rle.scenegen_rle4(rle.scenegen_default(64, 64, 64, 5))) as scene:
        n = rle.frame_workspace_bytes(endless)
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        with pytest.raises(rle.RLEError) as e:
            rle.render_frame(scene, cam, endless, ws, n, *outs[3])
        assert e.value.name == "RLE_ERR_INVALID_ARG"
        server = rle.Server(1 << 28, 1 << 18, max_frames_per_batch=8, max_samples=W)
        sid = server.add_scene(scene)
        server.pause(True)
        for k in range(3):
            server.submit(sid, cam, good, *outs[k])
            with pytest.raises(rle.RLEError) as e:
                server.submit(sid, cam, endless, *outs[3])
            assert e.value.name == "RLE_ERR_INVALID_ARG"
        server.pause(False)
        server.drain()
        done = server.poll()
        assert len(done) == 3 and all(d.status == 0 for d in done)
        server.destroy()
