"""CPU suite: memory that runs out while a format or a layout is built is an error of the call (or, for the layout, the templates' own
kernels), never the end of the process."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "alphasparse_b200")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("alloc") / "alloc_in_regions")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fopenmp", "-I/usr/local/cuda/include", os.path.join(HERE, "alloc_in_regions.cpp"), "-o", exe,
                    "-L" + PKG, "-l:libasp_b200.so", "-Wl,-rpath," + PKG], check=True)
    return exe


@pytest.mark.parametrize("part", ["layout", "validate", "K2", "K6", "K9", "B1", "D1"])
@pytest.mark.parametrize("mode", ["region", "any"])
def test_memory_runs_out(program, mode, part):
    r = subprocess.run([program, mode, part], capture_output=True, text=True, timeout=300, env=dict(os.environ, OMP_NUM_THREADS="4"))
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-500:])
    assert part + " built" in r.stdout
