"""The fixed-point EOS and geometry of the FMA and mixed builds at the bounds of what they
admit, against long double (fixed_bounds_selftest.cc)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def selftest(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("bounds") / "fixed_bounds_selftest")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fwrapv", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "lulesh_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "fixed_bounds_selftest.cc")], check=True)
    return exe


@pytest.mark.parametrize("what", ["expanding", "floor", "sound", "rates", "quotients"])
def test_bounds_against_extended_precision(selftest, what):
    r = subprocess.run([selftest, what], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
