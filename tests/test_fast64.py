"""The branch-free FP64 arithmetic of the geodesic integrator (so_fast64.cuh), on the host: division,
reciprocal and square root must round as the IEEE operators do (seeds up to 2^-19 off), a whole
Dormand-Prince attempt must return dp54()'s error, state and derivatives bit for bit, operands out of
range must be flagged, and the swept angle must be good to 1e-14 rad (the arguments' own rounding at
|dphi| <= 20 is 3.6e-15, the fits add 3e-16 of the angle, the chord 1e-15)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = tmp_path_factory.mktemp("fast64") / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I",
                    os.path.join(ROOT, "spacetime-optics_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "fast64_check.cpp")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    return {line.split()[0]: (int(line.split()[1]), int(line.split()[2]), float(line.split()[3]))
            for line in out if line}


@pytest.mark.parametrize("name", ["rcp", "div", "sqrt", "accept", "attempts", "notok", "flagged", "still", "nan"])
def test_rounds_as_ieee(rows, name):
    bad, n, _ = rows[name]
    assert n > 0 and bad == 0


def test_swept_angle(rows):
    assert rows["angle"][2] <= 1e-14
