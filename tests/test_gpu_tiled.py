"""GPU: the column-tiled layout that plan groups with scattered columns run (csrc/kernels_tiled.cu), against the CPU oracle at
the sizes where its tiles, slices and work shares end: columns that fill the last tile exactly, by one, or leave one over; rows
longer than a tile's piece limit; several sub-matrices in one group; x and y off 16-byte alignment; every clearing mode."""
import numpy as np
import pytest

import refdump
from alphasparse_b200 import capi, matrices as M, tuner

pytestmark = pytest.mark.gpu

TILE = {np.float32: 40672, np.float64: 20320}  # columns of a tile
NODES = {"K9": ["tlb_nnz 16"], "K10": ["tlb_nnz 7"], "K6": ["row_padding 32 1", "blb_row_evenly 32", "tlb_col_fixed 4"], "K4": ["wlb_col_fixed 64"],
         "K8": ["row_padding 4 1", "blb_row_evenly 4", "wlb_col_fixed 64"], "K7": ["blb_col_fixed 256"], "K2": ["row_padding 128 1", "blb_row_evenly 128", "tlb_row"],
         "K3": ["row_padding 32 1", "tlb_row"]}


def matrix(dtype, cols, seed, longest=70):
    rng = np.random.default_rng(seed)
    # just above what makes the layout the faster one
    lengths = rng.integers(40, longest, size=(4_000_000 if dtype is np.float32 else 9_000_000) // ((40 + longest) // 2))
    if longest == 71:  # a few hub rows: their pieces are summed in the warp before they reach y
        lengths[[0, 1, 777, -1]] = [cols // 2, 20_000, 3_000, 33]
    return M.from_row_lengths(lengths, cols, seed=seed, dtype=dtype)


@pytest.mark.parametrize("template,dtype,tiles,over,longest", [
    ("K9", np.float32, 3, 0, 71), ("K9", np.float64, 4, 1, 71), ("K10", np.float32, 3, -1, 71), ("K6", np.float32, 2, 1, 70), ("K6", np.float64, 5, 0, 70),
    ("K4", np.float32, 3, 1, 71), ("K8", np.float64, 4, -1, 70), ("K7", np.float32, 5, 7, 71), ("K2", np.float32, 3, 0, 70), ("K3", np.float64, 3, 1, 70)])
def test_tiled_group_matches_the_oracle(asp_ctx, template, dtype, tiles, over, longest):
    import torch

    m, x = matrix(dtype, tiles * TILE[dtype] + over, seed=tiles, longest=longest)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 1}]})
    assert g.layout_bytes() > 0, "the layout was not built for this matrix"
    y_ref, scale = refdump.csr_ref(m, x)
    for shift in (0, 1):  # x and y on and off 16-byte boundaries
        dx = torch.zeros(m.n_cols + shift, dtype=torch.from_numpy(x).dtype, device="cuda")
        dx[shift:] = torch.from_numpy(x).cuda()
        dy = torch.full((m.n_rows + 5 + shift,), 7.0, dtype=dx.dtype, device="cuda")
        for zero_y in (True, "auto"):
            torch.cuda.synchronize()
            g.spmv(dx[shift:].data_ptr(), dy[shift:].data_ptr(), zero_y)
            asp_ctx.synchronize()
            y = dy.cpu().numpy()
            refdump.assert_y(y[shift : shift + m.n_rows], y_ref, scale, m.values.dtype, f"{template} zero_y={zero_y} shift={shift}")
            assert (y[:shift] == 7).all() and (y[shift + m.n_rows :] == 7).all()  # nothing beside y
    g.close()
    own = fmt.upload(asp_ctx, layout="none")
    assert own.layout_bytes() == 0
    refdump.assert_y(own.spmv_host(x), y_ref, scale, m.values.dtype, f"{template} own kernel")
    own.close()
    fmt.close()


def test_tiled_group_of_sorted_strips_and_empty_rows(asp_ctx):
    rng = np.random.default_rng(8)
    lengths = np.concatenate([rng.integers(20, 100, size=30_000), rng.integers(200, 900, size=4_000), [30_000, 9_000]])
    rng.shuffle(lengths)
    lengths[rng.integers(0, lengths.size, size=500)] = 0  # rows that no kernel stores: zero when y is cleared
    m, x = M.from_row_lengths(lengths, 150_000, seed=8)
    sub = lambda t: {"graph": t, "nodes": NODES[t], "template": t, "threads": 128, "row_reduce": 1}
    from alphasparse_b200.graph import Matrix

    hm = Matrix.from_csr(m)
    cm = hm.dense("dense sort 1\ndense rowdiv_exp 128 4096 8\ndense compress")
    desc = {"dense": "dense sort 1 | dense rowdiv_exp 128 4096 8 | dense compress", "subs": [sub("K2" if cm.sub_rows(i)[3] <= 128 else "K6" if cm.sub_rows(i)[3] <= 1024 else "K7") for i in range(cm.n_subs)]}
    y_ref, scale = refdump.csr_ref(m, x)
    for layout in ("auto", "none"):
        fmt, g = tuner.build(asp_ctx, m, desc, layout)
        assert (g.layout_bytes() > 0) == (layout == "auto")
        assert g.launches() == (1 if layout == "auto" else len(desc["subs"]))
        refdump.assert_y(g.spmv_host(x), y_ref, scale, m.values.dtype, f"strips {layout}")
        g.close()
        fmt.close()
    cm.close()
    hm.close()


def exact(m, x):
    """(A x, |A| |x|) in the next longer type."""
    t = np.float64 if m.values.dtype == np.float32 else np.longdouble
    p = m.values.astype(t) * x.astype(t)[m.indices.view(np.int32)]
    return np.add.reduceat(p, m.indptr[:-1]), np.add.reduceat(np.abs(p), m.indptr[:-1])


@pytest.mark.parametrize("template,dtype,rows,lo,hi,cols", [
    ("K6", np.float32, 60_000, 40, 121, 1_000_000), ("K8", np.float64, 60_000, 40, 121, 1_000_000), ("K4", np.float64, 60_000, 40, 121, 100_000),
    ("K7", np.float32, 4_000, 1000, 3001, 1_000_000), ("K7", np.float64, 4_000, 1000, 3001, 1_000_000), ("K7", np.float64, 4_000, 1000, 3001, 100_000), ("K9", np.float32, 250_000, 4, 29, 1_000_000)])
def test_tiled_sums_are_as_near_to_the_exact_ones_as_the_templates(asp_ctx, template, dtype, rows, lo, hi, cols):
    """The layout adds a row up in other parts than the template's kernel, but with no larger error."""
    import torch

    rng = np.random.default_rng(rows)
    m, x = M.from_row_lengths(rng.integers(lo, hi, size=rows), cols, seed=rows, dtype=dtype)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 1}]})
    assert g.layout_bytes() > 0, "the layout was not built for this matrix"
    ref, scale = exact(m, x)
    dx = torch.from_numpy(x).cuda()
    far = []
    for zero_y in (True, False):  # the layout; the template's kernel, which adds to the zeros in y
        dy = torch.zeros(m.n_rows, dtype=dx.dtype, device="cuda")
        torch.cuda.synchronize()
        g.spmv(dx.data_ptr(), dy.data_ptr(), zero_y)
        asp_ctx.synchronize()
        d = dy.cpu().numpy().astype(ref.dtype) - ref
        far.append((float(np.sqrt((d * d).sum() / (ref * ref).sum())), float((np.abs(d) / scale).max())))
    assert far[0][0] <= 1.01 * far[1][0], far  # (the 2-norm repeats to a percent; the largest is one row's)
    assert far[0][1] <= 1.25 * far[1][1], far
    g.close()
    fmt.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_tiled_sums_are_one_call_s_own(asp_ctx, dtype):
    """Infinite sums leave nothing behind; calls of another context, of a graph and of the plan's own context give the same y."""
    import torch

    m, x = matrix(dtype, 3 * TILE[dtype], seed=3)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": "K9", "nodes": NODES["K9"], "template": "K9", "threads": 128, "row_reduce": 1}]})
    assert g.layout_bytes() > 0
    y_ref, scale = refdump.csr_ref(m, x)
    hit = np.bincount(np.repeat(np.arange(m.n_rows), m.row_lengths())[m.indices == 17], minlength=m.n_rows) > 0
    bad = x.copy()
    bad[17] = np.inf
    y = g.spmv_host(bad)
    assert np.isinf(y[hit]).all() and np.isfinite(y[~hit]).all()
    refdump.assert_y(g.spmv_host(x), y_ref, scale, m.values.dtype, "after an infinite x")
    bad[17] = np.nan
    assert np.isnan(g.spmv_host(bad)[hit]).all()
    refdump.assert_y(g.spmv_host(x), y_ref, scale, m.values.dtype, "after x that is no number")
    dx, dys = torch.from_numpy(x).cuda(), [torch.full((m.n_rows,), 7.0, dtype=torch.from_numpy(x).dtype, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    other = capi.Context(0)
    for _ in range(20):  # on two streams at once
        g.spmv(dx.data_ptr(), dys[0].data_ptr(), True)
        capi.check(capi.lib().asp_spmv(other.handle, g._plans, g.n, dx.data_ptr(), dys[1].data_ptr(), 1))
    other.synchronize()
    asp_ctx.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(asp_ctx.stream)):
        g.spmv(dx.data_ptr(), dys[2].data_ptr(), True)
    for _ in range(5):
        graph.replay()  # on torch's stream
        g.spmv(dx.data_ptr(), dys[0].data_ptr(), True)
    torch.cuda.synchronize()
    asp_ctx.synchronize()
    for y, what in zip(dys, ("own context", "another context", "graph")):
        refdump.assert_y(y.cpu().numpy(), y_ref, scale, m.values.dtype, what)
    del graph
    other.close()
    g.close()
    fmt.close()


def test_a_refused_tuning_call_keeps_the_layout(asp_ctx):
    m, x = matrix(np.float32, 3 * TILE[np.float32], seed=3)
    y_ref, scale = refdump.csr_ref(m, x)
    for template, vec in (("K9", 1), ("K4", 0), ("K2", 3), ("K2", 8)):
        fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 1}]})
        held = g.layout_bytes()
        assert held > 0
        with pytest.raises(capi.AspError):
            g.set_tuning(0, vec, 0)
        assert g.layout_bytes() == held
        refdump.assert_y(g.spmv_host(x), y_ref, scale, m.values.dtype, template)
        g.close()
        fmt.close()


@pytest.mark.parametrize("template", ["K2", "K3", "K6", "K8"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_results_repeat_bit_for_bit_without_the_layout(asp_ctx, template, dtype):
    m, x = matrix(dtype, 3 * TILE[dtype], seed=5)
    fmt, g = tuner.build(asp_ctx, m, {"dense": "dense compress", "subs": [{"graph": template, "nodes": NODES[template], "template": template, "threads": 128, "row_reduce": 1}]}, "none")
    y = g.spmv_host(x).copy()
    for _ in range(5):
        assert np.array_equal(g.spmv_host(x), y)
    g.close()
    fmt.close()


def test_an_unknown_layout_is_refused(asp_ctx):
    m, _ = M.uniform_random(300, 6, seed=1)
    from alphasparse_b200.graph import Matrix

    fmt = Matrix.from_csr(m).execute("dense compress\nsub all row_padding 32 1\nsub all tlb_row\nsub all template K3")
    descs = fmt.plan_descs()
    plans = (capi.C.c_void_p * len(descs))()
    with pytest.raises(capi.AspError):
        capi.check(capi.lib().asp_plan_group_create_with(asp_ctx.handle, (capi.PlanDesc * len(descs))(*descs), len(descs), 7, plans))
    fmt.close()


def test_the_layout_leaves_room_for_the_caller(asp_ctx):
    """On a device that is nearly full the group runs its templates' kernels."""
    import torch

    m, x = matrix(np.float32, 3 * TILE[np.float32], seed=3)
    y_ref, scale = refdump.csr_ref(m, x)
    desc = {"dense": "dense compress", "subs": [{"graph": "K9", "nodes": NODES["K9"], "template": "K9", "threads": 128, "row_reduce": 1}]}
    capi.device_trim(0)
    torch.cuda.empty_cache()
    full = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
    try:
        fmt, g = tuner.build(asp_ctx, m, desc)
        assert g.layout_bytes() == 0
        refdump.assert_y(g.spmv_host(x), y_ref, scale, m.values.dtype, "nearly full")
        g.close()
        fmt.close()
    finally:
        del full
        torch.cuda.empty_cache()
    fmt, g = tuner.build(asp_ctx, m, desc)
    assert g.layout_bytes() > 0
    assert 0.7 * g.format_bytes() < g.layout_bytes() < 1.3 * g.format_bytes()
    g.close()
    fmt.close()


@pytest.mark.parametrize("short,long,laid_out", [(2_000, 20, False), (5_000, 60, True)])
def test_small_groups_of_several_strips_keep_their_kernels(asp_ctx, short, long, laid_out):
    """Below 65,536 non-zeros every strip has the bits that it has with the others left out."""
    from alphasparse_b200.graph import Matrix

    rng = np.random.default_rng(short)
    m, x = M.from_row_lengths(np.concatenate([rng.integers(10, 30, size=short), rng.integers(500, 700, size=long)]), 50_000, seed=short)
    hm = Matrix.from_csr(m)
    cm = hm.dense("dense sort 1\ndense rowdiv_exp 128 4096 8\ndense compress")
    assert cm.n_subs > 1 and (m.nnz >= 65_536) == laid_out
    strip = lambda i, t: [f"sub {i} {n}" for n in NODES[t]] + [f"sub {i} template {t}"]
    templates = ["K2" if cm.sub_rows(i)[3] <= 128 else "K6" for i in range(cm.n_subs)]
    fmt = cm.execute("\n".join(l for i, t in enumerate(templates) for l in strip(i, t)))
    g = fmt.upload(asp_ctx)
    assert (g.layout_bytes() > 0) == laid_out
    y_ref, scale = refdump.csr_ref(m, x)
    y = g.spmv_host(x)
    refdump.assert_y(y, y_ref, scale, np.float32, "strips")
    if not laid_out:
        for i, t in enumerate(templates):
            part = cm.execute("\n".join(strip(i, t) + [f"sub {j} template EMPTY" for j in range(cm.n_subs) if j != i]))
            gp = part.upload(asp_ctx)
            assert gp.layout_bytes() == 0
            info = fmt.sub_info(i)
            rows = fmt.global_perm()[info.min_row : info.max_row + 1].astype(np.int64)
            assert np.array_equal(gp.spmv_host(x)[rows], y[rows])
            gp.close()
            part.close()
    g.close()
    fmt.close()
    cm.close()
    hm.close()


def test_strips_with_hub_rows_are_as_near_to_the_exact_sums(asp_ctx):
    """A small fp64 matrix: warps cut the long rows' pieces, two tiles only."""
    import torch

    rng = np.random.default_rng(9)
    m, x = M.from_row_lengths(np.concatenate([rng.integers(1, 12, size=30_000), rng.integers(200, 700, size=200), [9_000, 7_000, 5_000, 3_000]]), 30_000, seed=9, dtype=np.float64)
    from alphasparse_b200.graph import Matrix

    hm = Matrix.from_csr(m)
    cm = hm.dense("dense sort 1\ndense rowdiv_exp 128 4096 8\ndense compress")
    fmt = cm.execute("\n".join(l for i in range(cm.n_subs) for t in ["K2" if cm.sub_rows(i)[3] <= 128 else "K6" if cm.sub_rows(i)[3] <= 1024 else "K7"]
                               for l in [f"sub {i} {n}" for n in NODES[t]] + [f"sub {i} template {t}"]))
    g = fmt.upload(asp_ctx)
    assert g.layout_bytes() > 0
    ref, scale = exact(m, x)
    dx = torch.from_numpy(x).cuda()
    far = []
    for zero_y in (True, False):
        dy = torch.zeros(m.n_rows, dtype=dx.dtype, device="cuda")
        worst = 0.0
        for _ in range(4):  # (a few hub rows carry the norm: the order of their parts shows)
            dy.zero_()
            torch.cuda.synchronize()
            g.spmv(dx.data_ptr(), dy.data_ptr(), zero_y)
            asp_ctx.synchronize()
            d = dy.cpu().numpy().astype(ref.dtype) - ref
            worst += float(np.sqrt((d * d).sum() / (ref * ref).sum())) / 4
        far.append(worst)
    assert far[0] <= 1.1 * far[1], far
    g.close()
    fmt.close()
    cm.close()
    hm.close()
