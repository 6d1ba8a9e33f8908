"""The branch-free division and square root (so_fast64.cuh) where rounding is hardest, at results next to the
midpoint of two doubles (host build, seeds up to 2^-19 off): the square root rounds as the IEEE operator
does, and the quotient, whose correction uses a reciprocal that is not rounded itself, within one unit in the
last place, wrong in no more than one case in a hundred of these."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = tmp_path_factory.mktemp("midpoints") / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I",
                    os.path.join(ROOT, "spacetime-optics_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "fast64_midpoints.cpp")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    return {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out if line}


def test_quotients_next_to_midpoints(rows):
    bad, n, worst = rows["quotient"]
    assert n >= 1000000 and worst <= 1 and bad <= n // 100


def test_square_roots_next_to_midpoints(rows):
    bad, n, _ = rows["sqrt"]
    assert n >= 10000 and bad == 0
