"""GPU: the block-value kernel shares the slots of a block row among 1, 2, 4 or 8 warps by the size of the matrix; every way at
block-row counts that leave the last warp, the last CTA and the last lane's pair of rows partly empty, and slot counts that the
shares do not divide, against the CPU oracle."""
import numpy as np
import pytest

import refdump
from alphasparse_b200 import matrices as M
from alphasparse_b200.graph import Matrix
from test_block_value import blocky, spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("r,n,blocks", [
    (3, 31, 17), (3, 65, 27), (3, 33, 3),                 # eight warps a block row; one slot at most in some shares
    (3, 9_001, 8), (2, 1_501, 13), (4, 701, 11),          # four
    (3, 20_003, 12),                                      # two
    (3, 57_605, 12), (2, 1_501, 5), (4, 701, 5)])         # one
def test_shares_of_a_block_row(asp_ctx, r, n, blocks, dtype):
    if n > 2_000:
        m, x = M.block_fem(n, blocks, 300, seed=n, dtype=dtype)
    else:
        m, x = blocky(r, r, n, blocks, seed=n, dtype=dtype, band=min(n // 2, 300))
    fmt = Matrix.from_csr(m).execute(spec(r, r))
    g = fmt.upload(asp_ctx)
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(g.spmv_host(x), y_ref, scale, dtype, f"{n} block rows x {blocks}")
    g.close()
    fmt.close()
