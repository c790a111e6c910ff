"""CPU suite: a forked process builds formats after its parent has, without the threads that helped there."""
import subprocess
import sys

import pytest

SCRIPT = """
import os, sys, time, warnings
import numpy as np
from alphasparse_b200 import matrices as M
from alphasparse_b200.graph import Matrix

m, _ = M.from_row_lengths(np.full(int(sys.argv[1]), 8), 50_000, seed=1, dtype=np.float32)

def build():
    for nodes, template in (("row_padding 32 1\\nsub all tlb_row", "K3"), ("tlb_nnz 16", "K9"), ("block_value 2 2", "B1"),
                            ("row_padding 32 1\\nsub all blb_row_evenly 32\\nsub all tlb_col_fixed 4", "K6")):
        Matrix.from_csr(m).execute(f"dense compress\\nsub all {nodes}\\nsub all template {template}").close()

build()
warnings.simplefilter("ignore")
child = os.fork()
if child == 0:
    build()
    os._exit(7)
for _ in range(200):
    done, status = os.waitpid(child, os.WNOHANG)
    if done:
        sys.exit(0 if os.waitstatus_to_exitcode(status) == 7 else 1)
    time.sleep(0.05)
os.kill(child, 9)
os.waitpid(child, 0)
sys.exit(2)
"""


@pytest.mark.parametrize("rows", [500, 4_000, 30_000, 200_000])
def test_a_forked_process_builds_formats(rows):
    import os

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(rows)], cwd=root, capture_output=True, text=True, timeout=120, env=dict(os.environ, OMP_NUM_THREADS="4"))
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
