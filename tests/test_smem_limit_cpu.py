"""The kernels' shared-memory limits under contexts that are made on several threads
(csrc/smem_limit.h, tests/cxx/smem_limit_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pd-ipc-armadillodemo_gb300", "csrc")


def test_limits_are_never_lowered(tmp_path):
    from pdipc import build
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    exe = str(tmp_path / "smem_limit_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + CSRC, "-I" + cuda,
                    os.path.join(ROOT, "tests", "cxx", "smem_limit_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
