"""GPU: the kernels that take whole rows of the templates whose chunks of a row lie one after the other (csrc/kernels_rows.cu), against
the CPU oracle: rows that end on, before and behind a trip of a warp, a CTA or a row's lanes, the longest rows that they take and one element
more, empty rows, one row, sorted rows, every column width, x and y off 16-byte alignment, every clearing mode."""
import ctypes as C

import numpy as np
import pytest

import refdump
from alphasparse_b200 import capi, matrices as M, tuner

pytestmark = pytest.mark.gpu

NODES = {"K4": ["wlb_col_fixed 64"], "K7": ["blb_col_fixed 256"], "K8": ["row_padding 4 1", "blb_row_evenly 4", "wlb_col_fixed 64"],
         "K2": ["row_padding 128 1", "blb_row_evenly 128", "tlb_row"], "K3": ["row_padding 32 1", "tlb_row"],
         "K9": ["tlb_nnz 16"], "K9/5": ["tlb_nnz 5"], "K9/32": ["tlb_nnz 32"], "K10": ["tlb_nnz 8"], "K10/3": ["tlb_nnz 3"],
         "K6": ["row_padding 32 1", "blb_row_evenly 32", "tlb_col_fixed 4"]}
NO_LIST = {"K5": ["blb_row_evenly 64", "wlb_row_evenly 16", "tlb_col_fixed 4"]}


def matrix(lengths, cols, dtype):
    """Rows of exactly these lengths."""
    rng = np.random.default_rng(len(lengths))
    indices = np.concatenate([np.sort(rng.choice(cols, size=n, replace=False)) for n in lengths]).astype(np.uint32)
    values = rng.uniform(-1, 1, size=indices.size).astype(dtype)
    return M.CsrMatrix(len(lengths), cols, np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64), indices, values), rng.uniform(-1, 1, size=cols).astype(dtype)


EDGES = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 130, 255, 256, 257, 500]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("template,lengths,cols,dense,whole", [
    ("K4", EDGES + [512], 5_000, "dense compress", True),
    ("K4", EDGES + [513], 5_000, "dense compress", False),           # a warp takes 512 elements and no more
    ("K4", [3] * 1000 + [200], 256, "dense compress", True),         # 8-bit columns
    ("K4", [70], 90, "dense compress", True),
    ("K8", EDGES * 5, 60_000, "dense compress", True),               # 16-bit columns
    ("K8", EDGES + [0, 9, 0, 0, 77], 70_000, "dense compress", None),  # rows without elements
    ("K8", EDGES * 3, 2_000, "dense sort 1\ndense compress", True),
    ("K7", [1000, 1, 4095, 4096, 4097, 300, 16383], 40_000, "dense compress", True),
    ("K7", [16384, 3, 9000], 40_000, "dense compress", True),
    ("K7", [16385, 9000], 40_000, "dense compress", False),
    ("K7", [700] * 400 + [1023, 1024, 1025, 0], 70_000, "dense compress", None),  # (more rows than the device holds at once)
    ("K6", [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33] * 9, 3_000, "dense compress", True),
    ("K6", [1] * 500 + [4], 200, "dense compress", True),            # 8-bit columns, two lanes a row
    ("K6", [40, 41, 119, 120, 121] * 50, 70_000, "dense compress", True),
    ("K6", [120, 7, 64, 65] * 40, 9_000, "dense sort 1\ndense compress", True),
    ("K3", [9], 200, "dense compress", True),
    ("K3", [16] * 33, 3_000, "dense compress", True),                # four warps, one trip; a row in the second group
    ("K3", [17, 3, 1] * 32, 200, "dense compress", True),            # eight warps, 8-bit columns
    ("K3", [32, 8, 30] * 11, 70_000, "dense compress", True),
    ("K3", [33] * 31 + [64, 65, 129], 9_000, "dense compress", True),  # sixteen warps, one to three trips
    ("K3", [8] * 300, 9_000, "dense compress", False),               # the template's kernel has all of these in flight
    ("K2", [9] * 128 + [33] * 128 + [90] * 100, 9_000, "dense compress", True),  # strips of different lengths
    ("K2", [70, 12, 31, 1] * 65, 300, "dense sort 1\ndense compress", True),
    ("K9", [1], 3, "dense compress", True),
    ("K9", EDGES * 4, 9_000, "dense compress", True),
    ("K9/5", [1, 2, 3, 4, 5, 6] * 300 + [159, 160, 161], 9_000, "dense compress", True),
    ("K9/32", [4096, 1, 2, 3] + [30] * 90, 20_000, "dense compress", True),
    ("K9", [4097] + [30] * 90, 20_000, "dense compress", None),      # (with what fills the last warp)
    ("K10", [700, 3, 256, 1, 255] * 9, 3_000, "dense sort 1\ndense compress", True),
    ("K10/3", [7] * 100 + [57, 33, 32] * 3, 250, "dense compress", True),
    ("K6", [4] * 999 + [4 * 16 + 1], 3_000, "dense compress", False)])  # seventeen TLBs in a row, two lanes: eight trips and one
def test_whole_rows_match_the_oracle(asp_ctx, template, lengths, cols, dense, whole, dtype):
    import torch

    m, x = matrix(lengths, cols, dtype)
    fmt, g = tuner.build(asp_ctx, m, {"dense": dense.replace("\n", " | "), "subs": [{"graph": template, "nodes": NODES[template], "template": template.split("/")[0], "threads": 128, "row_reduce": 1}]})
    assert whole is None or (g.layout_bytes() == 0 and g.whole_rows() == whole)
    y_ref, scale = refdump.csr_ref(m, x)
    for shift in (0, 1):
        dx = torch.zeros(m.n_cols + shift, dtype=torch.from_numpy(x).dtype, device="cuda")
        dx[shift:] = torch.from_numpy(x).cuda()
        dy = torch.full((m.n_rows + 3 + shift,), 7.0, dtype=dx.dtype, device="cuda")
        modes = [True, "auto", False] if min(lengths) > 0 else [True]  # (rows that nobody stores are the caller's to clear)
        for zero_y in modes:
            if zero_y is False:  # the templates' own kernels, which add to y or overwrite it: both to a cleared one
                dy[shift : shift + m.n_rows] = 0
            torch.cuda.synchronize()
            g.spmv(dx[shift:].data_ptr(), dy[shift:].data_ptr(), zero_y)
            asp_ctx.synchronize()
            y = dy.cpu().numpy()
            refdump.assert_y(y[shift : shift + m.n_rows], y_ref, scale, dtype, f"{template} zero_y={zero_y} shift={shift}")
            assert (y[:shift] == 7).all() and (y[shift + m.n_rows :] == 7).all()  # nothing beside y
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("empty", [0, 20])
@pytest.mark.parametrize("zero_y", [True, "auto"])
def test_strips_by_whole_rows(asp_ctx, zero_y, empty, dtype):
    """Several sub-matrices with a kernel for whole rows each: all of them, some of them, one twice, one with its template's kernel."""
    import torch
    from alphasparse_b200.graph import Matrix

    lengths = np.random.default_rng(4).permutation([3] * 700 + [20] * 300 + [200] * 50 + [2000] * 5 + [0] * empty)
    m, x = matrix(list(lengths), 9_000, dtype)
    hm = Matrix.from_csr(m)
    cm = hm.dense("dense sort 1\ndense rowdiv_exp 128 4096 8\ndense compress")
    spec = []
    for i in range(cm.n_subs):
        t = "K2" if cm.sub_rows(i)[3] <= 128 else "K6" if cm.sub_rows(i)[3] <= 1024 else "K7"
        spec += [f"sub {i} {node}" for node in NODES[t]] + [f"sub {i} template {t}"]
    fmt = cm.execute("\n".join(spec))
    g = fmt.upload(asp_ctx)
    assert cm.n_subs > 1 and g.layout_bytes() == 0
    assert empty or all(capi.lib().asp_plan_whole_rows(g._plans[i]) for i in range(g.n))
    y_ref, scale = refdump.csr_ref(m, x)
    dx = torch.from_numpy(x).cuda()
    dy = torch.full((m.n_rows + 3,), 7.0, dtype=dx.dtype, device="cuda")
    if zero_y == "auto":
        dy[: m.n_rows] = 0
    torch.cuda.synchronize()
    for _ in range(2):
        g.spmv(dx.data_ptr(), dy.data_ptr(), zero_y)
    asp_ctx.synchronize()
    refdump.assert_y(dy.cpu().numpy()[: m.n_rows], y_ref, scale, dtype, "all strips")
    assert (dy[m.n_rows :] == 7).all()
    perm = fmt.global_perm()
    rows = [perm[fmt.sub_info(i).min_row : fmt.sub_info(i).max_row + 1].astype(np.int64) for i in range(g.n)]

    def call(which, mode):
        """y after a call of some plans of the group over a y of sevens"""
        dy[:] = 7
        torch.cuda.synchronize()
        plans = (C.c_void_p * len(which))(*[g._plans[i] for i in which])
        capi.check(capi.lib().asp_spmv(asp_ctx.handle, plans, len(which), C.c_void_p(dx.data_ptr()), C.c_void_p(dy.data_ptr()), mode))
        asp_ctx.synchronize()
        assert (dy[m.n_rows :] == 7).all()
        return dy.cpu().numpy()[: m.n_rows]

    for which in ([0], [g.n - 1], [g.n - 1, 0]):
        mine = np.concatenate([rows[i] for i in which])
        for mode in (1, 2):
            y = call(which, mode)
            refdump.assert_y(y[mine], y_ref[mine], scale[mine], dtype, f"plans {which}")
            others = np.setdiff1d(np.arange(m.n_rows), mine)
            assert (y[others] == 0).all() or (mode == 2 and (y[others] == 7).all())
    # a plan twice adds twice what it adds: the templates' kernels (the last strip's rows are added up or stored, as its template does)
    y = call([0, 0], 1)
    twice = 2 if fmt.plan_descs()[0].is_atom_add else 1
    refdump.assert_y(y[rows[0]], twice * y_ref[rows[0]], scale[rows[0]], dtype, "a plan twice")
    # one of them with its template's kernel
    capi.check(capi.lib().asp_plan_set_tuning(g._plans[g.n - 1], 0, 0))
    assert not capi.lib().asp_plan_whole_rows(g._plans[g.n - 1])
    refdump.assert_y(call(range(g.n), 1), y_ref, scale, dtype, "a tuned plan among others")
    g.close()
    fmt.close()
    cm.close()
    hm.close()


@pytest.mark.parametrize("template", ["K2", "K3", "K9"])
def test_a_tuned_plan_runs_its_own_kernel(asp_ctx, template):
    m, x = matrix([30, 40] * 100, 3_000, np.float32)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 1}]})
    assert g.whole_rows()
    y_ref, scale = refdump.csr_ref(m, x)
    capi.check(capi.lib().asp_plan_set_tuning(g._plans[0], 0, 0))
    assert not g.whole_rows()
    refdump.assert_y(g.spmv_host(x), y_ref, scale, np.float32, template)
    g.close()
    fmt.close()


@pytest.mark.parametrize("template", sorted(NODES))
def test_without_layouts_the_templates_kernels_run(asp_ctx, template):
    m, x = matrix([30, 40] * 100, 3_000, np.float32)
    desc = {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template.split("/")[0], "threads": 128, "row_reduce": 1}]}
    y_ref, scale = refdump.csr_ref(m, x)
    for layout in ("auto", "none"):
        fmt, g = tuner.build(asp_ctx, m, desc, layout)
        assert g.whole_rows() == (layout == "auto")
        refdump.assert_y(g.spmv_host(x), y_ref, scale, np.float32, f"{template} {layout}")
        g.close()
        fmt.close()


def strips_of(cm, templates):
    return [[f"sub {i} {node}" for node in (NODES | NO_LIST)[t]] + [f"sub {i} template {t}"] for i, t in enumerate(templates)]


@pytest.mark.parametrize("layout,short,long,templates,listed", [
    ("none", 20_000, 600, "K2 K6", 0),   # 800,000 stored elements
    ("none", 1_000, 30, "K2 K6", 0),
    ("auto", 1_000, 30, "K2 K6", 2),
    ("auto", 1_000, 30, "K2 K5", 1),     # one of the strips has no list
    ("auto", 1_000, 30, "K3 K8", 2),
    ("auto", 1_000, 30, "K9 K6", 2)])
def test_a_strip_has_the_same_bits_alone_and_in_its_group(asp_ctx, layout, short, long, templates, listed):
    from alphasparse_b200.graph import Matrix

    rng = np.random.default_rng(short)
    m, x = M.from_row_lengths(np.concatenate([rng.integers(10, 30, size=short), rng.integers(500, 700, size=long)]), 50_000, seed=short)
    hm = Matrix.from_csr(m)
    cm = hm.dense("dense sort 1\ndense rowdiv_exp 128 4096 8\ndense compress")
    strips = strips_of(cm, [templates.split()[cm.sub_rows(i)[3] > 128] for i in range(cm.n_subs)])
    assert cm.n_subs > 1 and (m.nnz < 65_536) == (short == 1_000)
    fmt = cm.execute("\n".join(sum(strips, [])))
    g = fmt.upload(asp_ctx, layout)
    assert g.layout_bytes() == 0
    y_ref, scale = refdump.csr_ref(m, x)
    y = g.spmv_host(x)
    refdump.assert_y(y, y_ref, scale, np.float32, "strips")
    whole = [bool(capi.lib().asp_plan_whole_rows(g._plans[i])) for i in range(g.n)]
    assert (sum(whole) > 0) == (listed > 0) and (listed == 1) == (0 < sum(whole) < g.n)
    for i, strip in enumerate(strips):
        part = cm.execute("\n".join(strip + [f"sub {j} template EMPTY" for j in range(cm.n_subs) if j != i]))
        gp = part.upload(asp_ctx, layout)
        assert bool(capi.lib().asp_plan_whole_rows(gp._plans[i])) == whole[i]
        info = fmt.sub_info(i)
        rows = fmt.global_perm()[info.min_row : info.max_row + 1].astype(np.int64)
        assert np.array_equal(gp.spmv_host(x)[rows], y[rows]), i
        gp.close()
        part.close()
    g.close()
    fmt.close()
    cm.close()
    hm.close()


def free_memory():
    import torch

    capi.check(capi.lib().asp_device_trim(0))
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("template", ["D1", "K3"])
def test_room_for_lists_goes_with_what_they_take(asp_ctx, template):
    """Plans that have none."""
    import torch

    m, x = M.laplacian_2d(600, seed=1, dtype=np.float64)
    desc = {"dense": "dense compress", "subs": [{"graph": template, "nodes": (NODES | {"D1": ["diag_value 64"]})[template], "template": template, "threads": 128, "row_reduce": 1}]}
    dx, dy = torch.from_numpy(x).cuda(), torch.full((m.n_rows,), 7.0, dtype=torch.from_numpy(x).dtype, device="cuda")
    before = free_memory()
    fmt, g = tuner.build(asp_ctx, m, desc)
    assert g.layout_bytes() == 0 and not g.whole_rows()
    assert before - free_memory() <= g.format_bytes() + (5 << 20)  # (allocations are in pieces of 2 MB)
    fmt_bytes = g.format_bytes()
    g.close()
    # room for the format and little more: the plan is made
    hold = torch.empty(free_memory() - fmt_bytes - (60 << 20), dtype=torch.uint8, device="cuda")
    try:
        g = fmt.upload(asp_ctx)
        g.spmv(dx.data_ptr(), dy.data_ptr(), True)
        asp_ctx.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(dy.cpu().numpy(), y_ref, np.maximum(scale, 1e-30), x.dtype, template)
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("template,rows,length", [("K7", 1_500, 2_000), ("K7", 3_000, 1_000), ("K4", 4_000, 500)])
def test_long_dense_rows_are_not_laid_out(asp_ctx, template, rows, length, dtype):
    """Rows of adjacent columns: the lanes of the column-tiled kernel would meet in one bank of shared memory."""
    rng = np.random.default_rng(rows)
    indices = (np.arange(rows, dtype=np.int64)[:, None] + np.arange(length)).reshape(-1).astype(np.uint32)
    m = M.CsrMatrix(rows, rows + length, np.arange(rows + 1, dtype=np.int64) * length, indices, rng.uniform(-1, 1, size=indices.size).astype(dtype))
    x = rng.uniform(-1, 1, size=m.n_cols).astype(dtype)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 1}]})
    assert g.whole_rows() and g.layout_bytes() == 0
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(g.spmv_host(x), y_ref, scale, dtype, template)
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("template", sorted(NODES))
def test_numbers_that_are_none(asp_ctx, template, dtype):
    """What is infinite or no number stays with the rows that have it, and a sum that passes the type's range is infinite."""
    m, x = matrix([30, 12, 1, 40, 33] * 40 + [300] * (template == "K7"), 3_000, dtype)
    if template == "K7":
        m, x = matrix([300, 700, 1000] * 20, 3_000, dtype)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template.split("/")[0], "threads": 128, "row_reduce": 1}]})
    assert g.whole_rows()
    y_ref, scale = refdump.csr_ref(m, x)
    hit = np.bincount(np.repeat(np.arange(m.n_rows), m.row_lengths())[m.indices == 17], minlength=m.n_rows) > 0
    assert 0 < hit.sum() < m.n_rows
    for what in (np.inf, -np.inf, np.nan):
        bad = x.copy()
        bad[17] = what
        y = g.spmv_host(bad)
        assert not np.isfinite(y[hit]).any() and (np.isnan(y[hit]).all() or not np.isnan(what))
        refdump.assert_y(y[~hit], y_ref[~hit], scale[~hit], dtype, f"beside {what}")
    # (the products stay in range, their sum does not)
    most = np.finfo(dtype).max
    big = M.CsrMatrix(m.n_rows, m.n_cols, m.indptr, m.indices, np.full(m.nnz, most / 4, dtype=dtype))
    f2, g2 = tuner.build(asp_ctx, big, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template.split("/")[0], "threads": 128, "row_reduce": 1}]})
    for sign in (1, -1):
        y = g2.spmv_host(np.full(m.n_cols, sign, dtype=dtype))
        assert (y[m.row_lengths() >= 5] == sign * np.inf).all() and np.isfinite(y[m.row_lengths() < 4]).all()
    for o in (g, fmt, g2, f2):
        o.close()


@pytest.mark.parametrize("template", sorted(NODES))
def test_whole_rows_in_a_graph_and_on_other_contexts(asp_ctx, template):
    """Lists hold no state."""
    import torch

    m, x = matrix([30, 40] * 100, 3_000, np.float64)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template.split("/")[0], "threads": 128, "row_reduce": 1}]})
    assert g.whole_rows()
    y_ref, scale = refdump.csr_ref(m, x)
    dx, dys = torch.from_numpy(x).cuda(), [torch.full((m.n_rows,), 7.0, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    other = capi.Context(0)
    for _ in range(20):
        g.spmv(dx.data_ptr(), dys[0].data_ptr(), True)
        capi.check(capi.lib().asp_spmv(other.handle, g._plans, g.n, dx.data_ptr(), dys[1].data_ptr(), 1))
    other.synchronize()
    asp_ctx.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(asp_ctx.stream)):
        g.spmv(dx.data_ptr(), dys[2].data_ptr(), True)
    for _ in range(5):
        graph.replay()
        g.spmv(dx.data_ptr(), dys[0].data_ptr(), True)
    torch.cuda.synchronize()
    asp_ctx.synchronize()
    for y, what in zip(dys, ("own context", "another context", "graph")):
        refdump.assert_y(y.cpu().numpy(), y_ref, scale, np.float64, what)
    del graph
    other.close()
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("rows,length,step,listed", [
    (20_000, 30, 1, True), (24_000, 30, 1, False), (24_000, 30, 4, False), (24_000, 30, 50, True),  # 0.64, 0.77 M stored, columns near one another or not
    (90_000, 8, 1, True), (3_000, 300, 1, True), (20_000, 80, 1, "fp64"), (9_000, 80, 1, True)])
def test_row_grouped_rows_near_one_another(asp_ctx, rows, length, step, listed, dtype):
    """Their strips stream faster from some size on: those plans have no list."""
    rng = np.random.default_rng(rows)
    indices = (np.arange(rows, dtype=np.int64)[:, None] + np.arange(length) * step).reshape(-1).astype(np.uint32)
    m = M.CsrMatrix(rows, rows + length * step, np.arange(rows + 1, dtype=np.int64) * length, indices, rng.uniform(-1, 1, size=indices.size).astype(dtype))
    x = rng.uniform(-1, 1, size=m.n_cols).astype(dtype)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": "K6", "nodes": NODES["K6"], "template": "K6", "threads": 128, "row_reduce": 4}]})
    assert g.layout_bytes() == 0 and g.whole_rows() == (dtype == np.float64 if listed == "fp64" else listed)
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(g.spmv_host(x), y_ref, scale, dtype, f"{rows} rows of {length}")
    g.close()
    fmt.close()


@pytest.mark.parametrize("template", ["K4", "K6"])
@pytest.mark.parametrize("rows,length", [(10_000, 80), (14_000, 80)])
def test_whole_rows_of_a_short_x_are_not_laid_out(asp_ctx, rows, length, template):
    """fp32, x of one tile: its gathers cost little, and the layout has little to stream."""
    m, x = matrix([length] * rows, rows, np.float32)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 4}]})
    assert g.whole_rows() and g.layout_bytes() == 0
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(g.spmv_host(x), y_ref, scale, np.float32, template)
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("zero_y", [True, "auto"])
def test_strips_with_and_without_lists_in_one_call(asp_ctx, zero_y, dtype):
    """A strip that adds to y and cannot have a list (a row of more than 16,384 elements, in chunks) beside two that have one."""
    import torch
    from alphasparse_b200.graph import Matrix

    m, x = matrix([20] * 300 + [17_000] + [600] * 10 + [20] * 200 + [18_001], 50_000, dtype)
    hm = Matrix.from_csr(m)
    cm = hm.dense("dense sort 1\ndense rowdiv_exp 128 4096 8\ndense compress")
    longest = [cm.sub_rows(i)[3] for i in range(cm.n_subs)]
    names = ["K2" if n <= 128 else "K6" if n <= 1024 else "K7" for n in longest]
    assert sorted(set(names)) == ["K2", "K6", "K7"] and m.nnz < 65_536
    fmt = cm.execute("\n".join(sum(strips_of(cm, names), [])))
    g = fmt.upload(asp_ctx)
    assert [bool(capi.lib().asp_plan_whole_rows(p)) for p in g._plans] == [n != "K7" for n in names]
    assert [bool(d.is_atom_add) for d in fmt.plan_descs()] == [n == "K7" for n in names]
    y_ref, scale = refdump.csr_ref(m, x)
    dx, dy = torch.from_numpy(x).cuda(), torch.full((m.n_rows + 3,), 7.0, dtype=torch.from_numpy(x).dtype, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        g.spmv(dx.data_ptr(), dy.data_ptr(), zero_y)
    asp_ctx.synchronize()
    refdump.assert_y(dy.cpu().numpy()[: m.n_rows], y_ref, scale, dtype, "strips")
    assert (dy[m.n_rows :] == 7).all()
    for o in (g, fmt, cm, hm):
        o.close()
