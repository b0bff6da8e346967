"""Index range of the fast builds' face states (csrc/cell_states.cuh)."""
import os
import subprocess

from conftest import PKG_DIR

HERE = os.path.dirname(os.path.abspath(__file__))


def test_face_states_read_inside_the_region(tmp_path):
    include = "/usr/local/cuda/include"
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-std=c++17", "-O0", "-fsanitize=address", "-I", include, "-I",
                           os.path.join(PKG_DIR, "csrc"), os.path.join(HERE, "cell_states_check.cpp"),
                           "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
