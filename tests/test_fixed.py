"""The fixed-point geometry and EOS of the FMA and mixed builds against the
same formulas in long double, the elements their formats refuse, and the strict
build's integer division and square root against the hardware's
(fixed_selftest.cc)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def selftest(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fixed") / "fixed_selftest")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fwrapv", "-ffp-contract=off", "-I" + os.path.join(ROOT, "lulesh_gb300", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "fixed_selftest.cc")], check=True)
    return exe


@pytest.mark.parametrize("what", ["forces", "kinematics", "eos", "sums", "exact", "elements", "refused"])
def test_fixed_point_against_extended_precision(selftest, what):
    r = subprocess.run([selftest, what], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
