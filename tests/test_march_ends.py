"""Rays that would march for ever are refused on the host: level distances that
doubling cannot move past z (0: a mip_distance of 1 with any pitch) and steps
too short for z to grow (z_far past 2^24 without a switch before).  Compiled for
the host, without a GPU, against the march's own loop."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "rle-based-voxel-raycasting_gb300" / "csrc"


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cuda = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = Path(cuda).resolve().parent.parent / "include"
    if shutil.which("g++") is None or not (include / "cuda_runtime_api.h").exists():
        pytest.skip("g++ or the CUDA headers not found")
    out = tmp_path_factory.mktemp("march") / "march_check"
    # the scene loader's entry points are not called: sections dropped by the linker
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-ffunction-sections", "-Wl,--gc-sections",
           "-I", str(ROOT / "include"), "-I", str(CSRC), "-I", str(include),
           str(ROOT / "tests" / "c" / "march_check.cpp"), *[str(CSRC / f) for f in ("frame.cpp", "raymap.cpp", "scene.cpp")],
           "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return out


@pytest.mark.parametrize("seed", [1, 2])
def test_endless_marches_are_refused(check, seed):
    r = subprocess.run([str(check), str(seed), "20000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    bad, ends, endless, zero, zero_launched, one, one_launched = map(int, r.stdout.split())
    assert bad == 0
    assert ends > 10000 and endless > 300
    assert (zero, zero_launched) == (-1, 0)  # RLE_ERR_INVALID_ARG, nothing launched
    assert (one, one_launched) == (0, 1)
