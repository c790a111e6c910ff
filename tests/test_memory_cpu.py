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


@pytest.mark.parametrize("part", ["ring", "threads", "no memory", "full device", "views"])
def test_copies_and_pools(program, part):
    r = subprocess.run([program, part], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-500:])
    assert part + ": ok" in r.stdout


def test_every_device_allocation_may_use_the_idle_memory():
    """cudaMalloc is called in one place, which gives idle blocks back when it fails."""
    src = os.path.join(os.path.dirname(HERE), "alphasparse_b200", "csrc")
    calls = [(f, line) for f in sorted(os.listdir(src)) if f.endswith((".cu", ".h")) for line in open(os.path.join(src, f)) if "cudaMalloc(" in line and "//" not in line.split("cudaMalloc(")[0]]
    assert {f for f, _ in calls} == {"memory.cu"} and len(calls) == 2, calls
