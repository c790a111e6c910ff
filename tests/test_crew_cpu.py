"""CPU suite: loops shared among a caller and helpers (csrc/host/crew.cpp): every piece once, whoever is there; by several callers at once,
inside of pieces, in forked processes, and where all helpers are held up."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", params=["", "thread"])
def program(request, tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("crew") / "crew")
    flags = ["-O2"] if not request.param else ["-O1", "-g", "-fsanitize=" + request.param]
    r = subprocess.run(["g++", "-std=c++17", "-fopenmp", "-pthread", *flags, os.path.join(HERE, "crew.cpp"), "-o", exe], capture_output=True, text=True)
    if r.returncode and request.param:
        pytest.skip("no sanitizer here: " + r.stderr[-200:])
    assert r.returncode == 0, r.stderr
    return exe, request.param


@pytest.mark.parametrize("part", ["cover", "callers", "held", "forked", "region"])
def test_shared_loops(program, part):
    exe, sanitizer = program
    if sanitizer and part in ("forked", "region"):
        pytest.skip("the sanitizer does not know OpenMP's barriers, nor threads after a fork")
    r = subprocess.run([exe, part], capture_output=True, text=True, timeout=300, env=dict(os.environ, TSAN_OPTIONS="exitcode=66"))
    if "FATAL: ThreadSanitizer" in r.stderr:
        pytest.skip(r.stderr[-200:])
    assert r.returncode == 0, (r.returncode, r.stdout[-500:], r.stderr[-3000:])
