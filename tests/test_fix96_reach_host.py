"""The potential's inverse distance of fixed-point positions (inv_distance_fix96 in
gravhopper_gb300/csrc/f64emu.cuh) at separations and softenings near 2^-31 of the box, the
shortest it takes, with the device's seed, whose range nothing checks.

Bound as in the whole box (below 1.25 half-ulps): a taken pair keeps its leading bit at 2^62
or at 2^60 of the sum of squares, and is off by no more units than any other."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("reach") / "fix96_reach_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "native", "fix96_reach_check.cpp")], check=True)
    return exe


@pytest.mark.parametrize("mode", range(3))
def test_taken_within_rounding_else_refused(checker, mode):
    n = 400_000
    r = subprocess.run([checker, str(n), str(mode), "3"], capture_output=True, text=True, timeout=300, check=True)
    taken, refused, worst, near = r.stdout.split()
    assert float(worst) < 1.25
    # everything from 2^-31 of the box on is taken, but for truncation at that very edge
    assert abs(int(taken) - int(near)) <= n // 100_000
    assert int(taken) + int(refused) == n and int(refused) > n // 4
