"""The tile partition of the persistent solve (csrc/tile_plan.cpp), checked on
the host against the tables it is built from: grids of many sizes and
numberings, several models, launch limits, both value sizes and summation
orders (tests/cxx/tile_plan_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pd-ipc-armadillodemo_gb300", "csrc")


def test_tile_plan_matches_the_host_tables(tmp_path):
    exe = str(tmp_path / "tile_plan_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, os.path.join(ROOT, "tests", "cxx", "tile_plan_check.cpp"),
                    os.path.join(CSRC, "tile_plan.cpp"), os.path.join(CSRC, "host_tables.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
