"""The work that programs have this renderer do, as cases that can be timed.

A case is a dict of plain values.  Every kind of case goes through the
package's public entry points, the way a user's program calls them:

  frame     render_frame: one camera to one screen (an interactive viewer)
  rays      raymap_build + render_rays + resolve with hit records: the drop-in
            for the reference's cuda_main_render2 and colorize pass, with
            picking
  batch     Batch.render: many cameras in one call
  serve     Server.submit for each request of a burst, then drain
  soft      soft_filter: the post-filter over a resolved frame
  encode    Scene.encode_on_device of a voxel volume, then rle_scene_copy_level
            of every level into the converter's own host buffers
  generate  Scene.generate_on_device, then the first frame of the session
  load      Scene.from_bytes of .rle4 bytes, then the first frame

Scenes, cameras and volumes come from the seed.  Scene grids, screen sizes
and poses follow the package's benchmark: fBm terrain with or without caves,
eyes 10-80 voxels above the ground, any yaw, pitch up to 30 degrees, samples
per column ray the next power of two of the width (or the width itself, the
library's default).
"""
import ctypes
import importlib.util
import math
import random
import struct
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parents[1] / "rle-based-voxel-raycasting_gb300"


def _package():
    if "rle_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("rle_gb300", PKG / "__init__.py",
                                                      submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["rle_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["rle_gb300"]


# Screen sizes of a mixed batch and of the requests a server gets, with the
# weights of the benchmark's two mixes.
BATCH_MIX = (((320, 240), 1), ((640, 480), 1), ((1280, 720), 1), ((1920, 1080), 1))
SERVE_MIX = (((256, 256), 4), ((640, 480), 3), ((1280, 720), 2), ((1920, 1080), 1))


# Words of a column that a converter's host buffers hold, on average.
COLUMN_WORDS = 80


def listed():
    return [
        # the smallest frame in use: a preview or an agent's view; a few
        # hundred column rays, so launches and one ray's latency count
        dict(name="frame_320x240", kind="frame", grid=512, height=256, caves=False, width=320, rows=240,
             samples="pow2", fov=90.0, mip=0),
        # an ordinary small viewer over plain terrain
        dict(name="frame_640x480", kind="frame", grid=512, height=256, caves=False, width=640, rows=480,
             samples="pow2", fov=90.0, mip=0),
        # the reference user's replacement calls on a laptop screen (1366 is
        # no multiple of a warp), with a hit record per sample and per pixel
        dict(name="rays_1366x768_hits", kind="rays", grid=1024, height=256, caves=True, width=1366, rows=768,
             samples="width", fov=90.0, mip=0),
        # the headline frame: 1080p over a 2048^2 cave scene
        dict(name="frame_1920x1080", kind="frame", grid=2048, height=256, caves=True, width=1920, rows=1080,
             samples="pow2", fov=90.0, mip=0),
        # the largest single frame: 4K, 75 degrees, near LOD switches, over
        # the largest scene
        dict(name="frame_3840x2160", kind="frame", grid=8192, height=512, caves=True, width=3840, rows=2160,
             samples="pow2", fov=75.0, mip=256),
        # offline or multi-user rendering: cameras at mixed resolutions, the
        # launch shape that the autotuner picks for throughput
        dict(name="batch_64_mixed", kind="batch", grid=2048, height=256, caves=True, frames=64, width=0, rows=0,
             lanes=16, per_frame=True, fov=90.0, mip=0),
        # eight 4K views per call with the batch's own defaults
        dict(name="batch_8_3840x2160", kind="batch", grid=4096, height=512, caves=True, frames=8, width=3840,
             rows=2160, lanes=0, per_frame=True, fov=75.0, mip=256),
        # a burst of requests to a server with two resident scenes
        dict(name="serve_48", kind="serve", grid=1024, height=256, caves=True, requests=48),
        # the display pass over a 1080p frame
        dict(name="soft_1920x1080", kind="soft", grid=1024, height=256, caves=True, width=1920, rows=1080),
        # a converter: coloured voxel volume on the device to an encoded scene
        # on the host
        dict(name="encode_512x256x512", kind="encode", grid=512, height=256, colours=True, levels=4),
        # the start of a session on generated terrain
        dict(name="generate_2048", kind="generate", grid=2048, height=256, caves=True, width=1280, rows=720),
        # the start of a session on an .rle4 file's bytes
        dict(name="load_512", kind="load", grid=512, height=256, caves=True, width=640, rows=480),
    ]


def draw(rng: random.Random):
    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def screen(lo, hi):
        w = log_uniform(lo, hi)
        return w, max(8, min(w, int(w * rng.uniform(0.4, 1.0))))

    kind = rng.choice(("frame", "frame", "frame", "rays", "batch", "batch", "serve", "soft", "encode", "generate",
                       "load"))
    grid = rng.choice((256, 512, 1024, 2048, 4096))
    height = rng.choice((128, 256, 512))
    caves = rng.random() < 0.7
    mip = rng.choice((0, 0, 256))
    fov = rng.choice((90.0, 90.0, 75.0, round(rng.uniform(45.0, 110.0), 1)))
    if kind in ("frame", "rays"):
        w, h = screen(64, 3840)
        return dict(kind=kind, grid=grid, height=height, caves=caves, width=w, rows=h,
                    samples=rng.choice(("pow2", "pow2", "width")), fov=fov, mip=mip)
    if kind == "batch":
        n = log_uniform(2, 96)
        w, h = screen(96, 1280) if rng.random() < 0.6 else (0, 0)
        n = min(n, 64) if w == 0 else max(2, min(n, 60_000_000 // (w * h)))
        return dict(kind=kind, grid=min(grid, 2048), height=height, caves=caves, frames=n, width=w, rows=h,
                    lanes=rng.choice((0, 16, 32)), per_frame=rng.random() < 0.75, fov=fov, mip=mip)
    if kind == "serve":
        return dict(kind=kind, grid=min(grid, 1024), height=256, caves=caves, requests=log_uniform(4, 64))
    if kind == "soft":
        w, h = screen(64, 2048)
        return dict(kind=kind, grid=min(grid, 1024), height=256, caves=caves, width=w, rows=h)
    if kind == "encode":
        return dict(kind=kind, grid=rng.choice((64, 128, 256, 512)), height=rng.randint(40, 300),
                    colours=rng.random() < 0.6, levels=rng.randint(1, 4))
    w, h = screen(160, 1280)
    if kind == "generate":
        return dict(kind=kind, grid=min(grid, 2048), height=min(height, 256), caves=caves, width=w, rows=h)
    return dict(kind=kind, grid=min(grid, 1024), height=height, caves=caves, width=w, rows=h)


# ------------------------------------------------------------------ inputs

def _scene_params(rle, case, seed, grid=None):
    n = grid or case["grid"]
    p = rle.scenegen_default(n, case["height"], n, seed, caves=case["caves"])
    if n == 8192:  # the large scene's denser caves (about 12 runs per column)
        p.cave_threshold = 0.25
        p.cave_period = 66.0
    return p


def _copy_level(rle, scene, mip, table, words=None):
    """rle_scene_copy_level into host arrays that the caller keeps."""
    at = [ctypes.c_void_p(a.ctypes.data) if a is not None else None for a in (table, words)]
    status = rle.library().rle_scene_copy_level(scene.handle, mip, *at)
    if status != 0:
        raise RuntimeError("rle_scene_copy_level: %d" % status)


def _column_tops(rle, scene):
    """Index of the first voxel of every column (z, x), counted from the top."""
    info = scene.info()
    table = np.empty((info.sz[0], info.sx[0], 2), np.uint32)
    _copy_level(rle, scene, 0, table)
    return (table[..., 1] >> 16) & 1023


def _cameras(rle, scene, rng, count, fov, lo=10.0, hi=80.0):
    info = scene.info()
    tops = _column_tops(rle, scene)
    sx, sy, sz = info.sx[0], info.sy[0], info.sz[0]
    cams = []
    for _ in range(count):
        x, z = rng.uniform(0, sx), rng.uniform(0, sz)
        ground = sy - int(tops[int(z) % sz, int(x) % sx])
        pitch = rng.uniform(1.0, 30.0) * rng.choice((-1.0, 1.0))
        cams.append(rle.camera(x, z, ground + rng.uniform(lo, hi), rng.uniform(0.0, 360.0), pitch, fov,
                               scene_height=sy))
    return cams


def _pow2_ceil(v):
    return 1 << max(3, (v - 1).bit_length())


def _view(rle, w, h, samples="pow2", mip=0):
    return rle.view_params(w, h, samples=_pow2_ceil(w) if samples == "pow2" else 0, mip_distance=mip)


def _screen(pixels):
    return (torch.empty(pixels, dtype=torch.int32, device="cuda"),
            torch.empty(pixels, dtype=torch.float32, device="cuda"))


def _frame_state(rle, st, scene, rng, case, samples="pow2"):
    st["cam"] = _cameras(rle, scene, rng, 1, case.get("fov", 90.0))[0]
    st["view"] = _view(rle, case["width"], case["rows"], case.get("samples", samples), case.get("mip", 0))
    st["ws"] = torch.empty(rle.frame_workspace_bytes(st["view"]), dtype=torch.uint8, device="cuda")
    st["colour"], st["depth"] = _screen(case["width"] * case["rows"])


def _mixed(mix, count):
    """`count` screen sizes of a mix, the same ones for every seed."""
    sizes, weights = zip(*mix)
    return random.Random(count).choices(sizes, weights, k=count)


def _rle4_bytes(scene):
    """The scene as .rle4 bytes: the file a user has on disk."""
    info = scene.info()
    out = [struct.pack("<i", info.nummaps)]
    for m in range(info.nummaps):
        _, words = scene.copy_level(m)
        out.append(struct.pack("<iiii", info.sx[m], info.sy[m], info.sz[m], words.size))
        out.append(words.tobytes())
    return b"".join(out)


def _volume(case, seed):
    """A voxel volume in the reference's Tree layout, bits and RGB565 colours:
    smooth ground with round caves, thin overhangs and a few loose blocks."""
    n, sy = case["grid"], case["height"]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def noise(shape, size):
        v = torch.rand((1, 1, *shape), generator=gen, device="cuda")
        mode = "bicubic" if len(shape) == 2 else "trilinear"
        return torch.nn.functional.interpolate(v, size=size, mode=mode, align_corners=False)[0, 0]

    cells = max(4, n // 48)
    ground = noise((cells, cells), (n, n)) * 0.6 + noise((4 * cells, 4 * cells), (n, n)) * 0.1 + 0.15
    y = torch.arange(sy, device="cuda").view(1, sy, 1)  # 0 = top
    solid = y >= (sy * (1.0 - ground)).view(n, 1, n)
    caves = noise((cells, max(2, sy // 24), cells), (n, sy, n))
    solid &= caves < 0.66
    solid |= caves < 0.02
    weights = 1 << torch.arange(8, device="cuda", dtype=torch.int32)
    bits = (solid.view(n, sy, n // 8, 8).to(torch.int32) * weights).sum(-1).to(torch.uint8).contiguous()
    colours = None
    if case["colours"]:
        colours = torch.randint(-32768, 32767, (n, sy, n), generator=gen, device="cuda", dtype=torch.int16)
    return bits, colours


def prepare(case, seed):
    rle = _package()
    rng = random.Random(seed * 7919 + 13)
    kind = case["kind"]
    st = {"rle": rle, "case": case, "kind": kind}
    if kind == "encode":
        st["bits"], st["colours"] = _volume(case, seed)
        st["levels"] = []
        for m in range(case["levels"]):  # host buffers for the largest scene the converter takes
            n = case["grid"] >> m
            st["levels"].append((np.zeros(2 * n * n, np.int32), np.zeros(COLUMN_WORDS * n * n, np.int16)))
        return st
    scene = rle.Scene.generate_on_device(_scene_params(rle, case, seed))
    if kind in ("frame", "rays"):
        st["scene"] = scene
        _frame_state(rle, st, scene, rng, case)
        if kind == "rays":
            words = rle.raybuf_words(rle.raymap_build(st["cam"], st["view"]))
            st["ws"] = None
            st["raybuf"] = torch.zeros(words, dtype=torch.int32, device="cuda")
            st["raydepth"] = torch.zeros(words, dtype=torch.float32, device="cuda")
            st["rayhit"] = torch.zeros(words, dtype=torch.int64, device="cuda")
            st["hit"] = torch.empty(case["width"] * case["rows"], dtype=torch.int64, device="cuda")
    elif kind == "batch":
        one = [(case["width"], case["rows"])] * case["frames"]
        sizes = one if case["width"] else _mixed(BATCH_MIX, case["frames"])
        cams = _cameras(rle, scene, rng, len(sizes), case["fov"])
        views = [_view(rle, w, h, "pow2", case["mip"]) for w, h in sizes]
        st["scene"] = scene
        st["colour"], st["depth"] = _screen(sum(w * h for w, h in sizes))
        st["frames"], at = [], 0
        for cam, view in zip(cams, views):
            n = view.width * view.height
            st["frames"].append(rle.frame_request(cam, view, st["colour"][at:at + n], st["depth"][at:at + n]))
            at += n
        st["batch"] = rle.Batch(len(sizes), rle.batch_words_needed(st["frames"]), max(v.samples for v in views))
        if case["lanes"] or not case["per_frame"]:
            st["batch"].set_tuning(1, case["lanes"] or 32, 1, 128, True, case["per_frame"])
    elif kind == "serve":
        scenes = [scene, rle.Scene.generate_on_device(_scene_params(rle, case, seed + 1, 2 * case["grid"]))]
        st["scenes"] = scenes
        st["server"] = rle.Server(hbm_budget_bytes=120 << 30, raybuf_words=32 << 20, max_frames_per_batch=64,
                                  max_inflight=3, max_samples=2048)
        ids = [st["server"].add_scene(s) for s in scenes]
        views = [_view(rle, w, h) for w, h in _mixed(SERVE_MIX, case["requests"])]
        st["colour"], st["depth"] = _screen(sum(v.width * v.height for v in views))
        pools = [_cameras(rle, s, rng, len(views), 90.0) for s in scenes]
        st["requests"], at = [], 0
        for k, view in enumerate(views):
            which, n = rng.randrange(len(scenes)), view.width * view.height
            st["requests"].append((ids[which], pools[which][k], view, st["colour"][at:at + n],
                                   st["depth"][at:at + n]))
            at += n
    elif kind == "soft":
        _frame_state(rle, st, scene, rng, case)
        rle.render_frame(scene, st["cam"], st["view"], st["ws"], st["ws"].numel(), st["colour"], st["depth"])
        torch.cuda.synchronize()
        st["ws"] = None
        st["out"] = torch.empty_like(st["colour"])
        scene.free()
    elif kind in ("generate", "load"):
        _frame_state(rle, st, scene, rng, case)
        if kind == "generate":
            st["params"] = _scene_params(rle, case, seed)
        else:
            st["bytes"] = _rle4_bytes(scene)
        scene.free()
    return st


def _first_frame(st, scene):
    info = scene.info()
    st["rle"].render_frame(scene, st["cam"], st["view"], st["ws"], st["ws"].numel(), st["colour"], st["depth"])
    scene.free()
    return {"words": [int(info.slab_words[m]) for m in range(info.nummaps)], "runs": int(info.run_headers),
            "voxels": int(info.surface_voxels), "colour": st["colour"], "depth": st["depth"]}


def run(st):
    rle, kind = st["rle"], st["kind"]
    if kind == "frame":
        rle.render_frame(st["scene"], st["cam"], st["view"], st["ws"], st["ws"].numel(), st["colour"], st["depth"])
        return st["colour"], st["depth"]
    if kind == "rays":
        rm = rle.raymap_build(st["cam"], st["view"])
        rle.render_rays(st["scene"], rm, st["raybuf"], st["raydepth"], st["rayhit"])
        rle.resolve(rm, st["raybuf"], st["raydepth"], st["colour"], st["depth"], st["rayhit"], st["hit"])
        return st["raybuf"], st["raydepth"], st["rayhit"], st["colour"], st["depth"], st["hit"]
    if kind == "batch":
        st["batch"].render(st["scene"], st["frames"])
        return st["colour"], st["depth"]
    if kind == "serve":
        server = st["server"]
        for request in st["requests"]:
            server.submit(*request)
        server.drain()
        for done in server.poll():
            if done.status != 0:
                raise RuntimeError("request failed: %d" % done.status)
        return st["colour"], st["depth"]
    if kind == "soft":
        rle.soft_filter(st["colour"], st["depth"], st["case"]["width"], st["case"]["rows"], st["out"])
        return st["out"]
    if kind == "encode":
        n, sy, levels = st["case"]["grid"], st["case"]["height"], st["case"]["levels"]
        with rle.Scene.encode_on_device(st["bits"], st["colours"], n, sy, n, levels) as scene:
            info = scene.info()
            for m, (table, words) in enumerate(st["levels"]):
                if info.slab_words[m] > words.size:
                    raise RuntimeError("level %d has %d words" % (m, info.slab_words[m]))
                _copy_level(rle, scene, m, table, words)
        return st["levels"]
    if kind == "generate":
        return _first_frame(st, rle.Scene.generate_on_device(st["params"]))
    return _first_frame(st, rle.Scene.from_bytes(st["bytes"]))


def work(case):
    """Bytes and operations of one pass.  A pixel costs its colour and depth
    written and one colour word of the scene read; what else of the scene a
    frame reads depends on the view and is not counted.  An encoded column
    costs its table entry and about eight slab words."""
    kind = case["kind"]
    pixels = case.get("width", 0) * case.get("rows", 0)
    if kind == "batch":
        pixels = case["frames"] * (pixels or sum(w * h for (w, h), _ in BATCH_MIX) // len(BATCH_MIX))
    if kind == "serve":
        total = sum(k for _, k in SERVE_MIX)
        pixels = case["requests"] * sum(w * h * k for (w, h), k in SERVE_MIX) // total
    if kind == "soft":  # 33 bilinear taps of 4 texels x 4 channels at most
        return {"bytes": 12 * pixels, "flops": 33 * 32 * pixels}
    columns = case["grid"] ** 2 * 4 // 3
    if kind == "encode":
        bits = case["grid"] ** 2 * case["height"] // 8
        return {"bytes": bits + columns * (8 + 16 + (8 if case["colours"] else 0)), "flops": 0}
    if kind == "rays":  # ray buffer, depth and hits of about 1.5 rays per pixel column
        samples = _pow2_ceil(case["width"]) if case["samples"] == "pow2" else case["width"]
        return {"bytes": pixels * (8 + 2 + 8) + case["width"] * 3 // 2 * samples * 16, "flops": 0}
    extra = columns * (8 + 16) if kind in ("generate", "load") else 0
    return {"bytes": 10 * pixels + extra, "flops": 0}


def exact(case, seed):
    """No value in 64 bits: which voxel a sample shows hangs on the single
    precision steps of the column walk, so colours, hits, scene words and the
    depths that go with them are held to equality instead."""
    return None
