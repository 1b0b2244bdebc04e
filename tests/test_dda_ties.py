"""The DDA's jump over steps where the two axes meet at equal distances, compiled
for the host and compared with the steps bit for bit: directions in small
whole-number ratios from eyes at multiples of 1/16 of a cell, whose ties come to
lie at the edges of the distances' binades."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "rle-based-voxel-raycasting_gb300" / "csrc"


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    out = tmp_path_factory.mktemp("ties") / "dda_ties_check"
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC),
           str(ROOT / "tests" / "c" / "dda_ties_check.cpp"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return out


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_jumps_equal_the_steps_at_ties(check, seed):
    r = subprocess.run([str(check), str(seed), "100000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    bad, edges, ties = map(int, r.stdout.split())
    assert bad == 0
    assert edges > 1000000 and ties > 50000  # ties at the first step out of place were compared
