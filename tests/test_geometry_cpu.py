"""The closest-point distances and the filters of csrc/geometry.cuh, compiled for the
host (tests/cxx/geometry_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pd-ipc-armadillodemo_gb300", "csrc")


def test_geometry_on_the_host(tmp_path):
    from pdipc import build
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    exe = str(tmp_path / "geometry_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, "-I" + cuda,
                    os.path.join(ROOT, "tests", "cxx", "geometry_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
