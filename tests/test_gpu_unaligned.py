"""GPU: x and y of a call may begin anywhere that their type may: templates that store several rows at once, off 16-byte boundaries."""
import numpy as np
import pytest

import refdump
from alphasparse_b200 import matrices as M, tuner

pytestmark = pytest.mark.gpu

NODES = {"K2": ["row_padding 128 1", "blb_row_evenly 128", "tlb_row"], "K3": ["row_padding 32 1", "tlb_row"], "B1": ["block_value 3 3"], "D1": ["diag_value 64"]}


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("template", ["K2", "K3", "B1", "D1"])
def test_vectors_off_their_alignment(asp_ctx, template, dtype):
    import torch

    if template == "B1":
        m, x = M.block_fem(500, 5, 100, seed=1, dtype=dtype)
    else:
        m, x = M.laplacian_2d(41, seed=1, dtype=dtype, grid_y=37)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 1}]}, "none")
    y_ref, scale = refdump.csr_ref(m, x)
    for shift in range(4):
        dx = torch.zeros(m.n_cols + shift, dtype=torch.from_numpy(x).dtype, device="cuda")
        dx[shift:] = torch.from_numpy(x).cuda()
        dy = torch.full((m.n_rows + 5 + shift,), 7.0, dtype=dx.dtype, device="cuda")
        torch.cuda.synchronize()
        g.spmv(dx[shift:].data_ptr(), dy[shift:].data_ptr(), "auto")
        asp_ctx.synchronize()
        y = dy.cpu().numpy()
        refdump.assert_y(y[shift : shift + m.n_rows], y_ref, scale, dtype, f"{template} shift={shift}")
        assert (y[:shift] == 7).all() and (y[shift + m.n_rows :] == 7).all()
    g.close()
    fmt.close()
