"""The tags of the words that the CTAs of the one-kernel decode exchange (csrc/decode_tags.h):
none is met twice, however long a process decodes."""
import os
import subprocess

from conftest import PKG_DIR

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_word_passes_as_a_later_layers(tmp_path):
    exe = str(tmp_path / "decode_tags_test")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror",
                    "-I", os.path.join(PKG_DIR, "csrc"),
                    os.path.join(HERE, "fake_cuda", "decode_tags_test.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
