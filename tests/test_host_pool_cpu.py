"""Host buffers of the format operators are kept for later use, 256 MB in all: what is pushed out must be out of use."""
import zlib

import numpy as np

from alphasparse_b200 import matrices as M
from alphasparse_b200.graph import Matrix


def lowered(m):
    hm = Matrix.from_csr(m)
    cm = hm.dense("dense compress")
    fmt = cm.execute("sub all row_padding 32 1\nsub all tlb_row\nsub all template K3")
    cm.close()
    hm.close()
    return fmt


def checksum(fmt):
    return [(name, zlib.adler32(np.ascontiguousarray(arr))) for name, (arr, *_) in fmt.arrays(0).items() if arr is not None]


def test_buffers_pushed_out_of_the_pool():
    small = M.from_row_lengths(np.full(30_000, 20), 40_000, seed=1, dtype=np.float32)[0]
    held = lowered(small)
    expect = checksum(held)
    for rows in (250_000, 330_000, 420_000):  # 40, 53 and 67 MB an array pair, several at a time
        m = M.from_row_lengths(np.full(rows, 20), 40_000, seed=rows, dtype=np.float32)[0]
        a, b = lowered(m), lowered(m)
        assert checksum(a) == checksum(b)
        a.close()
        b.close()
        again = lowered(small)
        assert checksum(again) == expect
        again.close()
    assert checksum(held) == expect
    held.close()
