"""The codes with which all products are exact (csrc/exact_codes.h), against the rule itself on
every code of x."""
import os
import subprocess

from conftest import PKG_DIR

HERE = os.path.dirname(os.path.abspath(__file__))


def test_codes_of_exact_products(tmp_path):
    exe = str(tmp_path / "exact_codes_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror",
                    "-I", os.path.join(PKG_DIR, "csrc"),
                    os.path.join(HERE, "fake_cuda", "exact_codes_test.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
