"""The fixed-point interaction factor m (|d|^2 + eps^2)^(-3/2) of the FP64 tree walk
(mass_inv_cube in gravhopper_gb300/csrc/f64emu.cuh), built for the host.

Bound: one rounding (2^-53) after truncations of at most 10 units in the 60-bit sum of
squares (2^-56.6, times 3/2), 2 units each in the residual and three products of at
least 58 bits (2^-57 each) and the omitted cubic term (2^-58): below 1.25 half-ulps, a
half-ulp being at most 2^-53 of the value."""
import shutil
import subprocess
import os

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("walk") / "walk_factor_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "native", "walk_factor_check.cpp")], check=True)
    return exe


@pytest.mark.parametrize("mode", range(7))
def test_factor_within_rounding_or_refused(checker, mode):
    n = 600_000
    r = subprocess.run([checker, str(n), str(mode), "5"], capture_output=True, text=True, timeout=300, check=True)
    taken, refused, worst = r.stdout.split()
    if mode == 6:  # out of range: the walk's FP64 operations take these
        assert int(taken) == 0 and int(refused) == n
    else:
        assert int(taken) == n and float(worst) < 1.25
