"""GPU: host calls of the diagonal-value template, whose rows run as soon as their x has arrived and go to the host from the kernel: around
the sizes of a piece of x, diagonals that reach back, ahead, far ahead or not at all, more rows than columns and fewer, x and y page-locked or not."""
import ctypes as C

import numpy as np
import pytest

import refdump
from alphasparse_b200 import capi, matrices as M
from alphasparse_b200.graph import Matrix

pytestmark = pytest.mark.gpu

PIECE = 896 << 10


def banded(n_rows, n_cols, offsets, seed, dtype):
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n_rows, dtype=np.int64), len(offsets))
    c = r + np.tile(np.sort(np.array(offsets, dtype=np.int64)), n_rows)
    keep = (c >= 0) & (c < n_cols)
    indptr = np.concatenate([[0], np.cumsum(np.bincount(r[keep], minlength=n_rows))]).astype(np.int64)
    values = rng.uniform(-1, 1, size=int(keep.sum())).astype(dtype)
    return M.CsrMatrix(n_rows, n_cols, indptr, c[keep].astype(np.uint32), values), rng.uniform(-1, 1, size=n_cols).astype(dtype)


def tall(n_rows, n_cols, seed, dtype):
    """Rows of two elements all over x: few diagonals would not hold them."""
    rng = np.random.default_rng(seed)
    c = np.stack([np.arange(n_rows) % (n_cols - 1), np.arange(n_rows) % (n_cols - 1) + 1], 1)
    return M.CsrMatrix(n_rows, n_cols, np.arange(n_rows + 1, dtype=np.int64) * 2, c.reshape(-1).astype(np.uint32), rng.uniform(-1, 1, size=2 * n_rows).astype(dtype)), rng.uniform(-1, 1, size=n_cols).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("rows,cols,offsets", [
    (1, 1, [0]), (7, 7, [-1, 0, 1]), (1000, 1003, [-1, 0, 3]),
    ("piece", 0, [-3, 0, 2]), ("piece*3/2", -1, [-300, 0, 300]), ("piece*3/2", 0, [-300, 0, 300]), ("piece*3/2", 1, [-1, 0, 1]),
    ("piece*4", 5, [0]), ("piece*4", 0, [-70000, -5, 0]), ("piece*4", -3, [-1, 0, 200000]), ("piece*5", 130000, [0, 130000]),
    ("piece*9", 1, [-2048, -1, 0, 1, 2048])])
def test_host_call_matches_the_oracle(asp_ctx, rows, cols, offsets, dtype):
    import torch

    es = np.dtype(dtype).itemsize
    n = eval(rows.replace("piece", str(PIECE)).replace("/", "//")) // es if isinstance(rows, str) else rows
    m, x = banded(n if isinstance(rows, str) else rows, n + cols if isinstance(rows, str) else cols, offsets, 3, dtype)
    fmt = Matrix.from_csr(m).execute("dense compress\nsub all diag_value 64\nsub all template D1")
    g = fmt.upload(asp_ctx)
    y_ref, scale = refdump.csr_ref(m, x)
    xp = torch.from_numpy(x).pin_memory().numpy()
    for name, hx in (("pageable", x), ("pinned", xp)):
        for again in range(2):  # (a second call finds the buffers as the first left them)
            refdump.assert_y(g.spmv_host(hx), y_ref, scale, dtype, f"{name} x, page-locked y, call {again}")
        y = np.full(m.n_rows, 7, dtype=dtype)  # pageable
        capi.check(capi.lib().asp_spmv_host(asp_ctx.handle, g._plans, g.n, C.c_void_p(hx.ctypes.data), C.c_void_p(y.ctypes.data)))
        refdump.assert_y(y, y_ref, scale, dtype, f"{name} x, pageable y")
    # nothing beside y
    yp = torch.full((m.n_rows + 9,), 7.0, dtype=torch.from_numpy(x).dtype).pin_memory()
    capi.check(capi.lib().asp_spmv_host(asp_ctx.handle, g._plans, g.n, C.c_void_p(x.ctypes.data), C.c_void_p(yp.data_ptr() + 3 * es)))
    refdump.assert_y(yp.numpy()[3 : 3 + m.n_rows], y_ref, scale, dtype, "page-locked y off its alignment")
    assert (yp[:3] == 7).all() and (yp[3 + m.n_rows :] == 7).all()
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("spec,threads", [("diag_value 64", "D1"), ("row_padding 32 1|tlb_row", "K3"), ("tlb_nnz 8", "K9")])
@pytest.mark.parametrize("rows,cols", [(5, 8), (96, 99), (1001, 1004), (40_000, 40_003), (60_001, 60_004), (250_000, 250_003), (60_000, 900), (530_000, 900), (1_060_000, 900)])
def test_pipelined_calls_around_a_short_x(asp_ctx, rows, cols, spec, threads, dtype):
    """x in one piece or in several, y from the kernels or by copies, page-locked or not, with chunks that read to the end of x or not."""
    import torch
    from alphasparse_b200 import tuner

    m, x = banded(rows, cols, [-2, 0, 3], 5, dtype) if cols > rows else tall(rows, cols, 5, dtype)
    if cols < rows and threads == "D1":
        pytest.skip("no diagonals")
    desc = {"dense": "dense compress", "subs": [{"graph": threads, "nodes": spec.split("|"), "template": threads, "threads": 128, "row_reduce": 1}]}
    chunks = tuner.build_row_chunks(asp_ctx, m, desc, 3, align=32)
    y_ref, scale = refdump.csr_ref(m, x)
    xp = torch.from_numpy(x).pin_memory()
    for pinned in (True, False):
        y = torch.full((rows + 2,), 7.0, dtype=xp.dtype)
        y = y.pin_memory() if pinned else y
        for _ in range(2):
            capi.spmv_host_pipelined(asp_ctx, [c[1:] for c in chunks], xp.data_ptr(), y.data_ptr())
        refdump.assert_y(y.numpy()[:rows], y_ref, scale, dtype, f"{threads} pinned={pinned}")
        assert (y[rows:] == 7).all()
    for fmt, g, *_ in chunks:
        g.close()
        fmt.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shift", [-4096, -1, 0, 1, 200_000])
def test_x_and_y_in_one_buffer(asp_ctx, shift, dtype):
    """Rows are stored while later x is on its way: not into what has yet to be read."""
    import torch

    n = 4 * PIECE // np.dtype(dtype).itemsize
    m, x = banded(n, n, [-1, 0, 1], 3, dtype)
    fmt = Matrix.from_csr(m).execute("dense compress\nsub all diag_value 64\nsub all template D1")
    g = fmt.upload(asp_ctx)
    y_ref, scale = refdump.csr_ref(m, x)
    both = torch.zeros(n + abs(shift), dtype=torch.from_numpy(x).dtype).pin_memory()
    hx, hy = both[max(0, -shift) :][:n], both[max(0, shift) :][:n]
    for _ in range(2):
        hx.copy_(torch.from_numpy(x))
        capi.check(capi.lib().asp_spmv_host(asp_ctx.handle, g._plans, g.n, C.c_void_p(hx.data_ptr()), C.c_void_p(hy.data_ptr())))
        refdump.assert_y(hy.numpy(), y_ref, scale, dtype, f"y {shift} behind x")
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bytes_of_chunks", [[(3 << 19) - 128, 3 << 19, (3 << 19) + 128], [3 << 20, 640, 2 << 20], [64 << 10, 5 << 20, 1 << 20]])
def test_pipelined_calls_with_long_chunks(asp_ctx, bytes_of_chunks, dtype):
    """Chunks of diagonal values of 1.5 MB and more go to page-locked y from the kernel, shorter ones by copies, in one call."""
    import torch

    es = np.dtype(dtype).itemsize
    rows = sum(bytes_of_chunks) // es
    m, x = banded(rows, rows, [-300, 0, 1, 2000], 5, dtype)
    y_ref, scale = refdump.csr_ref(m, x)
    made, chunks, lo = [], [], 0
    for n in bytes_of_chunks:
        hi = lo + n // es
        sub = m.row_slice(lo, hi)
        fmt = Matrix.from_csr(sub).execute("dense compress\nsub all diag_value 64\nsub all template D1")
        made.append((fmt, fmt.upload(asp_ctx)))
        chunks.append((made[-1][1], lo, hi, int(sub.indices.max()) + 1))
        lo = hi
    xp = torch.from_numpy(x).pin_memory()
    for pinned, shift in ((True, 0), (True, 1), (False, 0)):
        y = torch.full((rows + 4,), 7.0, dtype=xp.dtype)
        y = y.pin_memory() if pinned else y
        for _ in range(2):
            capi.spmv_host_pipelined(asp_ctx, chunks, xp.data_ptr(), y[shift:].data_ptr())
        refdump.assert_y(y.numpy()[shift : shift + rows], y_ref, scale, dtype, f"pinned={pinned} shift={shift}")
        assert (y[:shift] == 7).all() and (y[shift + rows :] == 7).all()
    for fmt, g in made:
        g.close()
        fmt.close()
