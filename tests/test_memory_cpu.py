"""CPU suite: the copies and the pools of csrc/memory.cu on a CUDA runtime of the host (fake_runtime.cpp)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("memory") / "fake_runtime")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fopenmp", "-I/usr/local/cuda/include", os.path.join(HERE, "fake_runtime.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("part", ["ring", "no memory"])
def test_copies_and_pools(program, part):
    r = subprocess.run([program, part], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-500:])
    assert part + ": ok" in r.stdout
