"""CPU suite: which plans have lists of their rows, and what those take (csrc/host/row_lists.cpp) by itself (row_lists.cpp)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "alphasparse_b200")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("rows") / "row_lists")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fopenmp", "-I/usr/local/cuda/include", os.path.join(HERE, "row_lists.cpp"), "-o", exe,
                    "-L" + PKG, "-l:libasp_b200.so", "-Wl,-rpath," + PKG], check=True)
    return exe


@pytest.mark.parametrize("part", ["limits", "empty"])
def test_lists(program, part):
    r = subprocess.run([program, part], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-500:])
