"""A launch does not depend on what else the process has launched: batches and
frames of few samples and small blocks, made or drawn in between, leave those of
many samples and large blocks as they are."""
from __future__ import annotations

import threading

import pytest

pytestmark = pytest.mark.gpu

W, H = 64, 48


@pytest.fixture(scope="module")
def scene(rle, torch_cuda):
    s = rle.Scene.from_bytes(rle.scenegen_rle4(rle.scenegen_default(64, 64, 64, 5, caves=True)))
    yield s
    s.free()


def _camera(rle):
    return rle.camera(30.0, 21.0, 60.0, 20.0, -12.0, scene_height=64)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("hits", [False, True])
def test_a_smaller_batch_in_between(rle, torch_cuda, scene, graph, hits):
    torch = torch_cuda

    def make(samples, threads):
        outs = [torch.zeros(W * H, dtype=torch.int32, device="cuda"), torch.zeros(W * H, device="cuda")]
        frames = [rle.frame_request(_camera(rle), rle.view_params(W, H, samples=samples), *outs)]
        b = rle.Batch(1, rle.batch_words_needed(frames), samples, with_hits=hits)
        b.set_tuning(1, 32, 1, threads, graph, 0)
        return b, frames, outs

    large, frames, large_outs = make(16384, 128)
    colour = large_outs[0]
    large.render(scene, frames)
    torch.cuda.synchronize()
    want = colour.clone()
    small, small_frames, small_outs = make(8, 32)
    small.render(scene, small_frames)
    colour.zero_()
    large.render(scene, frames)
    torch.cuda.synchronize()
    assert torch.equal(colour, want)
    small.free()
    large.free()
    del small_outs  # written by the small batch until here


def test_frames_of_many_sizes_from_many_threads(rle, torch_cuda, scene):
    torch = torch_cuda
    failed = []

    def draw(samples):
        try:
            view = rle.view_params(W, H, samples=samples)
            n = rle.frame_workspace_bytes(view)
            ws = torch.empty(n, dtype=torch.uint8, device="cuda")
            colour = torch.empty(W * H, dtype=torch.int32, device="cuda")
            depth = torch.empty(W * H, dtype=torch.float32, device="cuda")
            stream = torch.cuda.Stream()
            for i in range(1500):
                rle.render_frame(scene, _camera(rle), view, ws, n, colour, depth, stream=stream.cuda_stream)
                if i % 64 == 63:
                    stream.synchronize()
            stream.synchronize()
        except Exception as e:  # noqa: BLE001 -- any error of a thread fails the test
            failed.append((samples, e))

    threads = [threading.Thread(target=draw, args=(s,)) for s in (64, 16384, 128, 8192)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
