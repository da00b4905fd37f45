"""The FP64 tree walk's factor for massless particles (zero_mass_inv_cube in
gravhopper_gb300/csrc/f64emu.cuh), which keeps them off the FP64 pipe, built for the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_taken_where_a_mass_is(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "zero_mass_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "native", "zero_mass_check.cpp")], check=True)
    r = subprocess.run([exe, "400000", "2"], capture_output=True, text=True, timeout=300, check=True)
    taken, refused, wrong = map(int, r.stdout.split())
    assert wrong == 0 and taken > 200_000 and refused > 20_000
