"""The host's side of state uploads and downloads (csrc/host_copy.h): what a download
does to the caller's array before the copy must leave its contents, since the copy may
fail (tests/cxx/host_copy_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pd-ipc-armadillodemo_gb300", "csrc")


def test_copies_and_mapped_pages(tmp_path):
    exe = str(tmp_path / "host_copy_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "cxx", "host_copy_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
