"""The potential's inverse distance of 96-bit fixed-point positions (inv_distance_fix96 in
gravhopper_gb300/csrc/f64emu.cuh), built for the host.

Bound: one rounding (2^-53); differences off by 2 units, at least 2^30 units below the
leading bit kept (2^-61 of the distance); at most 10 units in the 60-bit sum of squares
(2^-56.7, halved by the root); 2 units each in the residual (2^-59) and the series
(2^-61): below 1.25 half-ulps."""
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
    exe = str(tmp_path_factory.mktemp("fix96") / "fix96_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "native", "fix96_check.cpp")], check=True)
    return exe


@pytest.mark.parametrize("mode", range(7))
def test_inverse_distance_within_rounding_or_refused(checker, mode):
    n = 500_000
    r = subprocess.run([checker, str(n), str(mode), "9"], capture_output=True, text=True, timeout=300, check=True)
    taken, refused, worst = r.stdout.split()
    if mode == 6:
        assert int(taken) == 0
    else:
        assert float(worst) < 1.25
        assert int(refused) == 0 or mode == 2 and int(refused) < n // 4
