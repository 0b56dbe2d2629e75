"""The page-locked staging of the host-pointer calls (csrc/host_stage.h) against a fake
runtime whose copies run as late as they may: slots, pieces, page-locked memory, and what a
call that fails half way leaves to the next one."""
import os
import subprocess

from conftest import PKG_DIR

HERE = os.path.dirname(os.path.abspath(__file__))


def test_host_stage_with_late_copies(tmp_path):
    exe = str(tmp_path / "host_stage_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fopenmp", "-Wall", "-Wextra", "-Werror",
                    "-I", os.path.join(HERE, "fake_cuda"), "-I", os.path.join(PKG_DIR, "csrc"),
                    os.path.join(HERE, "fake_cuda", "host_stage_test.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
