"""CPU suite: rows or warp-level blocks are shared out among the threads, whichever leaves none of them with nearly everything."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "alphasparse_b200")


def test_rows_or_blocks(tmp_path):
    exe = str(tmp_path / "wlb_rows")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(HERE, "wlb_rows.cpp"), "-o", exe, "-L" + PKG, "-l:libasp_b200.so", "-Wl,-rpath," + PKG], check=True)
    assert subprocess.run([exe], timeout=60).returncode == 0
