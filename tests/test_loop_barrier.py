"""The many-cycle launches' barrier counters over long simulations (bsim_b200/csrc/loop_barrier.h)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("barrier") / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror",
                    os.path.join(ROOT, "tests", "cpp", "loop_barrier_check.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("launches,cycles", [(1, 1), (1000, 4096), (20000000, 4096), (20000000, 1000), (3000000000, 1)])
def test_arrivals_stay_below_the_error_bits(check, launches, cycles):
    r = subprocess.run([check, str(launches), str(cycles)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
