"""Building the tile partition with a failing allocation: no plan or an exception the C
boundary turns into a status, never an abort (tests/cxx/tile_plan_alloc_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pd-ipc-armadillodemo_gb300", "csrc")


def test_failing_allocations_do_not_end_the_process(tmp_path):
    exe = str(tmp_path / "tile_plan_alloc_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "cxx", "tile_plan_alloc_check.cpp"),
                    os.path.join(CSRC, "tile_plan.cpp"), os.path.join(CSRC, "host_tables.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout + out.stderr)
