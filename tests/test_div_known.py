"""The division by a known divisor, over every mantissa of the dividend: the soft
filter's 255, and widths and heights of screens from the smallest to the largest."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "rle-based-voxel-raycasting_gb300" / "csrc"
DIVISORS = [255, 8, 9, 31, 100, 479, 480, 720, 1023, 1080, 1366, 1920, 2047, 2160, 3840, 8191, 16383, 16384]


def test_every_mantissa(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = tmp_path / "div_known_check"
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC),
           str(ROOT / "tests" / "c" / "div_known_check.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe), *map(str, DIVISORS)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["0", str(len(DIVISORS) << 23)]
