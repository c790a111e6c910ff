"""CPU suite: the column-tiled layout's host side (csrc/host/tiled_build.cpp) by itself (tiled_layout.cpp)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "alphasparse_b200")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("tiled") / "tiled_layout")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fopenmp", "-I/usr/local/cuda/include", os.path.join(HERE, "tiled_layout.cpp"), "-o", exe,
                    "-L" + PKG, "-l:libasp_b200.so", "-Wl,-rpath," + PKG], check=True)
    return exe


def run(program, *args, threads=4):
    r = subprocess.run([program, *map(str, args)], capture_output=True, text=True, timeout=300, env=dict(os.environ, OMP_NUM_THREADS=str(threads)))
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-500:])
    return r.stdout


def test_units_keep_to_32_bit_offsets(program):
    run(program, "fit")


@pytest.mark.parametrize("threads", [1, 3, 4, 16])
def test_the_choice_of_units_does_not_depend_on_the_threads(program, threads):
    for seed in (1, 2):
        run(program, "choice", seed, threads=threads)


@pytest.mark.parametrize("mode", ["y", "sums", "both"])
def test_units_hold_the_matrix(program, mode):
    run(program, "units", mode)


@pytest.mark.parametrize("threads", [1, 4])
def test_warps_of_a_cta_in_fp64(program, threads):
    run(program, "warps", threads=threads)
