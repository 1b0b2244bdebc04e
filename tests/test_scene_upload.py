"""A loaded scene is complete when the loader returns: frames run on streams that
do not wait for the default stream, on which the loader uploads.  Run on a CUDA
runtime of host memory, in which what is not waited for has not arrived."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "rle-based-voxel-raycasting_gb300" / "csrc"


@pytest.mark.parametrize("size,levels", [((8, 64, 8), 1), ((64, 64, 64), 4)])
@pytest.mark.parametrize("fails", [0, 1])
def test_loader_waits_for_its_upload(rle, tmp_path, size, levels, fails):
    cuda = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = Path(cuda).resolve().parent.parent / "include"
    if shutil.which("g++") is None or not (include / "cuda_runtime_api.h").exists():
        pytest.skip("g++ or the CUDA headers not found")
    p = rle.scenegen_default(*size, 7)
    p.nummaps, p.base_period = levels, 8
    data = tmp_path / "scene.rle4"
    data.write_bytes(rle.scenegen_rle4(p))
    exe = tmp_path / "upload_check"
    cmd = ["g++", "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(CSRC), "-I", str(include),
           str(ROOT / "tests" / "c" / "upload_check.cpp"), str(CSRC / "scene.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe), str(data), str(fails)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    status, on_the_way, scene = map(int, r.stdout.split())
    assert on_the_way == 0
    assert (status == 0, scene) == ((False, 0) if fails else (True, 1))  # a wait that fails is reported
