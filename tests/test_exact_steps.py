"""The closed forms of the kernels' chains of float additions -- the fill's
accumulators and the DDA's events -- against the plain loops they stand for:
the header the kernels include, compiled for the host and compared bit for bit
on random and on awkward inputs (ties, exact powers of two, sums that fall
through binades or change sign, subnormals, infinities, NaN; rays along an
axis to the last bit, eyes at negative coordinates, level switches)."""
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
    out = tmp_path_factory.mktemp("steps") / "exact_steps_check"
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC),
           str(ROOT / "tests" / "c" / "exact_steps_check.cpp"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return out


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_closed_forms_equal_the_loops(check, seed):
    r = subprocess.run([str(check), str(seed), "400000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    bad_acc, bad_steady, bad_dda, steady, placed = map(int, r.stdout.split())
    assert (bad_acc, bad_steady, bad_dda) == (0, 0, 0)
    assert steady > 50000 and placed > 8000 * 60 * 32 // 2  # the closed form is what was compared
