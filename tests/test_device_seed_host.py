"""The host checks of the fixed-point pair factors (gravhopper_gb300/csrc/f64emu.cuh) built as
the device builds them, without the range check on the seed's residual that host builds
keep: an input that this check would refuse has to be refused, or right, without it.
Bounds as in the checks themselves: below 1.25 half-ulps."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def programs(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = {}
    for name in ("fix96_check", "walk_factor_check"):
        out[name] = str(tmp_path_factory.mktemp("seed") / name)
        subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-DGH_EMU_DEVICE_SEED", "-o", out[name],
                        os.path.join(HERE, "native", name + ".cpp")], check=True)
    return out


@pytest.mark.parametrize("mode", range(7))
@pytest.mark.parametrize("name", ["fix96_check", "walk_factor_check"])
def test_right_or_refused(programs, name, mode):
    n = 300_000
    r = subprocess.run([programs[name], str(n), str(mode), "4"], capture_output=True, text=True, timeout=300, check=True)
    taken, refused, worst = r.stdout.split()
    assert float(worst) < 1.25 and int(taken) + int(refused) == n
    if mode == 6:  # all out of range
        assert int(taken) == 0
    else:
        assert int(refused) == 0 or name == "fix96_check" and mode == 2 and int(refused) < n // 1000
