"""GPU: results in recycled page-locked memory, device memory of plans used again, and SpMVs that leave the clearing of y out
because the kernel stores every row."""
import numpy as np
import pytest

import refdump
from alphasparse_b200 import matrices as M, tuner

pytestmark = pytest.mark.gpu


def desc(template, nodes, dense="dense compress"):
    return {"dense": dense, "subs": [{"graph": template, "nodes": nodes, "template": template, "threads": 128, "row_reduce": 1}]}


def test_results_that_are_held_keep_their_values(asp_ctx):
    m, x = M.laplacian_2d(200, 1, grid_y=150)  # 240 KB of y: page-locked
    fmt, g = tuner.build(asp_ctx, m, desc("D1", ["diag_value 64"]))
    y_ref, scale = refdump.csr_ref(m, x)
    held = [g.spmv_host(x * k) for k in range(4)]
    view = held[2][10:20]
    del held[2]  # its buffer lives on in the view
    later = [g.spmv_host(x * k) for k in range(5, 9)]
    for k, y in zip((0, 1, 3, 5, 6, 7, 8), held + later):
        refdump.assert_y(y, k * y_ref, np.maximum(k, 1) * scale, m.values.dtype, f"{k} x")
    assert np.allclose(view, 2 * y_ref[10:20])
    g.close()
    fmt.close()


def test_plans_made_and_destroyed_in_turn(asp_ctx):
    kept = []
    for k, n in enumerate((40, 300, 41, 300, 1000, 299, 300)):  # blocks of freed plans are taken by others, of about their size
        m, x = M.laplacian_2d(n, k, grid_y=50, dtype=np.float32)
        fmt, g = tuner.build(asp_ctx, m, desc("K3", ["row_padding 32 1", "tlb_row"]))
        y_ref, scale = refdump.csr_ref(m, x)
        kept.append((g, fmt, x, y_ref, scale))
        if k % 2:
            kept.pop(0)[0].close()
        for g2, _, x2, r2, s2 in kept:
            refdump.assert_y(g2.spmv_host(x2), r2, s2, np.float32, f"mesh {n}")
    for g, fmt, *_ in kept:
        g.close()
        fmt.close()


@pytest.mark.parametrize("template,nodes", [("K2", ["row_padding 128 1", "blb_row_evenly 128", "tlb_row"]), ("K3", ["row_padding 32 1", "tlb_row"]),
                                            ("K6", ["row_padding 32 1", "blb_row_evenly 32", "tlb_col_fixed 2"]), ("B1", ["block_value 3 3"]), ("D1", ["diag_value 64"])])
@pytest.mark.parametrize("dense", ["dense compress", "dense sort 1\ndense compress"])
def test_y_needs_no_clearing_where_every_row_is_stored(asp_ctx, template, nodes, dense):
    import torch

    m, x = M.block_fem(1_001, 9, 100, seed=5) if template == "B1" else M.laplacian_2d(77, 3, grid_y=53)
    if "sort" in dense:
        if template in ("B1", "D1"):
            pytest.skip("these templates keep the order of the rows")
        keep = np.arange(m.n_rows) % 5 != 0  # rows without non-zeros: no kernel stores them
        lengths = np.where(keep, m.row_lengths(), 0)
        m, x = M.from_row_lengths(lengths, m.n_cols, seed=2, dtype=np.float64)
    fmt, g = tuner.build(asp_ctx, m, desc(template, nodes, dense.replace("\n", " | ")))
    dx = torch.from_numpy(x).cuda()
    dy = torch.full((m.n_rows,), 9.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g.spmv(dx.data_ptr(), dy.data_ptr(), True)
    asp_ctx.synchronize()
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(dy.cpu().numpy(), y_ref, scale, np.float64, template)
    g.close()
    fmt.close()


@pytest.mark.parametrize("template", ["K9", "K10"])
@pytest.mark.parametrize("s", [1, 3, 4, 5, 11, 16, 40])
@pytest.mark.parametrize("empty", ["none", "some", "last"])
def test_csr5_like_rows_left_uncleared(asp_ctx, template, s, empty):
    """Rows that lie inside one thread's or one block's share are stored, only the shared ones are cleared before."""
    import torch

    rng = np.random.default_rng(s)
    lengths = rng.integers(1, 12, 5_003)
    lengths[[0, 2_000, 5_002]] = 900  # shared by several threads and blocks
    if empty == "some":
        lengths[rng.integers(1, 5_002, 700)] = 0
    elif empty == "last":
        lengths[-300:] = 0
    m, x = M.from_row_lengths(lengths, 4_096, seed=s, dtype=np.float32)
    fmt, g = tuner.build(asp_ctx, m, desc(template, [f"tlb_nnz {s}"]))
    dx = torch.from_numpy(x).cuda()
    dy = torch.full((m.n_rows,), 9.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        g.spmv(dx.data_ptr(), dy.data_ptr(), True)
    asp_ctx.synchronize()
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(dy.cpu().numpy(), y_ref, scale, np.float32, f"{template} {s} {empty}")
    g.close()
    fmt.close()


def test_idle_memory_is_given_back(asp_ctx):
    import torch
    from alphasparse_b200 import capi

    m, x = M.from_row_lengths(np.full(200_000, 40), 200_000, seed=4, dtype=np.float64)  # 100 MB of plan
    fmt, g = tuner.build(asp_ctx, m, desc("K3", ["row_padding 32 1", "tlb_row"]))
    held = g.format_bytes() + g.layout_bytes()
    g.close()
    fmt.close()
    before = torch.cuda.mem_get_info()[0]
    capi.device_trim(0)
    assert torch.cuda.mem_get_info()[0] >= before + held * 0.9
    with pytest.raises(capi.AspError):
        capi.device_trim(1000)


def test_host_calls_on_pageable_buffers(asp_ctx):
    """asp_spmv_host on arrays of the caller's own: x and y go through the pinned ring, which starts at another place each time."""
    from alphasparse_b200 import capi

    cases = []
    for rows in (65_535, 65_536, 65_537, 300_001, 4_500_000):  # y of 256 KB and an element around, no multiple of a piece, more than the ring
        lengths = np.full(rows, 2)
        m, _ = M.from_row_lengths(lengths, rows, seed=rows % 97, dtype=np.float32)
        fmt, g = tuner.build(asp_ctx, m, desc("K3", ["row_padding 32 1", "tlb_row"]))
        cases.append((m, fmt, g))
    rng = np.random.default_rng(1)
    for k in range(12):
        m, _, g = cases[k % len(cases)]
        x = rng.uniform(-1, 1, m.n_cols).astype(np.float32)
        y = np.full(m.n_rows + 2, 7, dtype=np.float32)
        y_ref, scale = refdump.csr_ref(m, x)
        capi.check(capi.lib().asp_spmv_host(asp_ctx.handle, g._plans, g.n, x.ctypes.data, y[1:].ctypes.data))
        x[:] = np.nan  # the caller's again
        refdump.assert_y(y[1:-1], y_ref, scale, np.float32, f"call {k}")
        assert y[0] == 7 and y[-1] == 7
    for _, fmt, g in cases:
        g.close()
        fmt.close()
