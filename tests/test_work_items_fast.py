"""The material phase's work items for the builds with the integer EOS
(work_items_fast_selftest.cc)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_work_items_of_the_integer_eos(tmp_path):
    exe = str(tmp_path / "work_items_fast")
    csrc = os.path.join(ROOT, "lulesh_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + csrc,
                    "-I" + os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "work_items_fast_selftest.cc"),
                    os.path.join(csrc, "lg_problem.cc")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
