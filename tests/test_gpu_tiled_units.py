"""GPU: the column-tiled layout of rows with few elements in a tile, against the CPU oracle: in units (fp32; csrc/kernels_tiled.cu,
k_tiled_units), where units and lanes end: rows that go on into the next lanes and units, lanes without a row's start, last units that are full,
by one or all but; rows added up in y, as 64-bit sums, and both; empty rows; infinite x; x and y off 16-byte alignment. The same matrices in
fp64 have slices. Which of them a matrix has is asserted: another one would be another kernel's test."""
import numpy as np
import pytest

import refdump
from alphasparse_b200 import matrices as M, tuner

pytestmark = pytest.mark.gpu

K9, K6 = ["tlb_nnz 32"], ["row_padding 32 1", "blb_row_evenly 32", "tlb_col_fixed 4"]


FP64 = {"direct": {"slices", "y"}, "sums": {"slices", "sums"}, "both": {"slices", "y", "sums"}}


def lengths(kind, rng):
    if kind == "direct":  # at most as many parts as the template adds in sequence (32): 15 tiles
        return rng.integers(20, 61, size=150_000)
    if kind == "sums":  # more than the 8 that this template allows
        return rng.integers(40, 121, size=60_000)
    # both, with rows of many units: rows enough for clearing y to be less than sums for all of them
    n = rng.integers(15, 31, size=750_000)
    n[[0, 1, 77_777, -1]] = [30_000, 257, 9_000, 256]
    return n


@pytest.mark.parametrize("kind,template,nodes", [("direct", "K9", K9), ("sums", "K6", K6), ("both", "K9", K9)])
@pytest.mark.parametrize("dtype,cols", [(np.float32, 600_000), (np.float64, 300_001)])
@pytest.mark.parametrize("empty", [0, 40])
def test_units_match_the_oracle(asp_ctx, kind, template, nodes, dtype, cols, empty):
    import torch

    rng = np.random.default_rng(empty)
    n = lengths(kind, rng)
    if empty:
        n[rng.integers(2, n.size - 1, size=empty)] = 0
    m, x = M.from_row_lengths(n, cols, seed=7, dtype=dtype)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": nodes, "template": template, "threads": 128, "row_reduce": 1}]})
    assert g.layout_form() == ({"units", *{"direct": ["y"], "sums": ["sums"], "both": ["y", "sums"]}[kind]} if dtype is np.float32 else FP64[kind])
    y_ref, scale = refdump.csr_ref(m, x)
    for shift in (0, 1):
        dx = torch.zeros(m.n_cols + shift, dtype=torch.from_numpy(x).dtype, device="cuda")
        dx[shift:] = torch.from_numpy(x).cuda()
        dy = torch.full((m.n_rows + 5 + shift,), 7.0, dtype=dx.dtype, device="cuda")
        torch.cuda.synchronize()
        for _ in range(3):
            g.spmv(dx[shift:].data_ptr(), dy[shift:].data_ptr(), True)
        asp_ctx.synchronize()
        y = dy.cpu().numpy()
        refdump.assert_y(y[shift : shift + m.n_rows], y_ref, scale, m.values.dtype, f"{kind} shift={shift}")
        assert (y[:shift] == 7).all() and (y[shift + m.n_rows :] == 7).all()
    hit = np.bincount(np.repeat(np.arange(m.n_rows), m.row_lengths())[m.indices == 17], minlength=m.n_rows) > 0
    bad = x.copy()
    bad[17] = np.inf
    y = g.spmv_host(bad)
    assert np.isinf(y[hit]).all() and np.isfinite(y[~hit]).all()
    bad[17] = np.nan
    y = g.spmv_host(bad)
    assert np.isnan(y[hit]).all() and np.isfinite(y[~hit]).all()
    refdump.assert_y(g.spmv_host(x), y_ref, scale, m.values.dtype, "after infinite x")
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("over", [0, 1, 255])
def test_last_units_of_the_tiles(asp_ctx, dtype, over):
    """Every tile holds full units and `over` elements: a row has four elements in each of the tiles, the last one `over` more."""
    tile, rows = (40672, 81_920) if dtype is np.float32 else (20320, 122_880)
    tiles = 12
    rng = np.random.default_rng(over)
    cols = [np.arange(tiles)[:, None] * tile + np.sort(rng.integers(0, tile, size=(rows, tiles, 4)), 2)]
    n = np.full(rows, 4 * tiles)
    last = np.sort(np.arange(tiles)[:, None] * tile + rng.integers(0, tile, size=(tiles, 4 + over)), 1)  # of the last row
    n[-1] = last.size
    cols = np.concatenate([cols[0][:-1].reshape(-1), last.reshape(-1)]).astype(np.uint32)
    m = M.CsrMatrix(rows, tiles * tile, np.concatenate([[0], np.cumsum(n)]).astype(np.int64), cols, rng.standard_normal(cols.size).astype(dtype))
    x = rng.standard_normal(m.n_cols).astype(dtype)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": "K9", "nodes": K9, "template": "K9", "threads": 128, "row_reduce": 1}]})
    assert ("units" if dtype is np.float32 else "slices") in g.layout_form()
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(g.spmv_host(x), y_ref, scale, m.values.dtype, f"over {over}")
    g.close()
    fmt.close()


@pytest.mark.parametrize("seed", [1, 2])
def test_rows_over_several_lanes_are_whole(asp_ctx, seed):
    """Small whole numbers, of which every sum is exact: a sum that lacks what other lanes hold of its row, or has it twice, differs. Runs of 1
    to 9 elements, some of hundreds, begin and end at every place of a lane."""
    tile, rows, tiles = 40672, 60_000, 16
    rng = np.random.default_rng(seed)
    runs = rng.integers(1, 10, size=(rows, tiles))
    runs[rng.integers(0, rows, size=300), rng.integers(0, tiles, size=300)] = rng.integers(30, 700, size=300)
    first = (np.arange(tiles) * tile + rng.integers(0, tile // 2, size=(rows, tiles))).reshape(-1)
    begin = np.concatenate([[0], np.cumsum(runs.reshape(-1))])
    at = np.arange(begin[-1]) - np.repeat(begin[:-1], runs.reshape(-1))
    cols = (np.repeat(first, runs.reshape(-1)) + at * 13).astype(np.uint32)
    m = M.CsrMatrix(rows, tiles * tile, np.concatenate([[0], np.cumsum(runs.sum(1))]).astype(np.int64), cols, rng.integers(-9, 10, size=cols.size).astype(np.float32))
    x = rng.integers(-9, 10, size=m.n_cols).astype(np.float32)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": "K9", "nodes": K9, "template": "K9", "threads": 128, "row_reduce": 1}]})
    assert "units" in g.layout_form()
    want = np.add.reduceat(m.values.astype(np.float64) * x[cols], m.indptr[:-1]).astype(np.float32)
    for _ in range(5):
        assert (g.spmv_host(x) == want).all()
    g.close()
    fmt.close()
