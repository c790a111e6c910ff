"""The work whose speed this repository answers for: y = A x over uploaded formats, and the calls around it.

Every case is a matrix of one of the shapes that the benchmark and the tests use, the graph that the search picks for such
a matrix (or one of the graphs it chooses among), and the call a program makes with it. Matrices, values and vectors are
made from the seed on the GPU; the sizes of the listed cases are those of the benchmark's configurations where a plan can be
built for them in a second or two, and smaller ones of the same shape where it cannot.

    rowgroup   uniformly random rows, a few non-zeros each: a small system in a loop; the call is as long as its launch
    diag       variable-coefficient 5-point stencil, stored by diagonals (fp64 solver)
    ell        the same stencil in the reference's own ELL-like format, odd grid
    block      finite elements with three unknowns per node, dense 3 x 3 blocks
    sell       the same matrix in the SELL-like format (search without the block operator)
    powerlaw   rows of Zipf-distributed length, random columns: CSR5-like format
    graph      x <- A x on an R-MAT graph with renumbered vertices, several iterations a pass, the native loop
    medium     rows of 40 to 120 non-zeros: row-grouped, warp-per-chunk and shared-memory warp formats
    long       rows of 1000 to 3000 non-zeros: a CTA per row chunk
    split      skewed rows, sorted and cut into strips with a format each: several kernels per SpMV
    host       x and y in host memory: the plain call, or the pipelined one on pinned buffers
    build      a matrix assembled anew: CSR in host memory -> format -> device -> first y
"""
from __future__ import annotations

import numpy as np
import torch

from alphasparse_b200 import capi, matrices_gpu, tuner
from alphasparse_b200.graph import Matrix
from alphasparse_b200.matrices import CsrMatrix

F32, F64 = "f32", "f64"


def listed():
    return [
        # 4096 rows, Poisson(16) a row: the benchmark's smallest configuration, an SpMV inside a small iterative solver
        {"name": "rowgroup-4096", "kind": "rowgroup", "rows": 4096, "mean": 16.0, "dtype": F32},
        # the benchmark's Laplacian mesh: one operator application of a fp64 solver
        {"name": "diag-2048x2048", "kind": "diag", "nx": 2048, "ny": 2048, "dtype": F64},
        # an odd mesh in fp32 (smoother of a mixed-precision multigrid): rows do not fill the last tile, x is never aligned
        {"name": "ell-1801x1603", "kind": "ell", "nx": 1801, "ny": 1603, "dtype": F32},
        # 3-D elasticity, 27 nodes a row, fp64
        {"name": "block-98304", "kind": "block", "nodes": 98304, "blocks": 27, "dtype": F64},
        # a finite-element matrix of the same kind that is stored without its blocks
        {"name": "sell-65537", "kind": "sell", "nodes": 65537, "blocks": 27, "dtype": F64},
        # the benchmark's power-law configuration: random columns over an x of 34 MB
        {"name": "powerlaw-8388608", "kind": "powerlaw", "rows": 8_388_608, "tlb": 16, "staged": True, "warp_reduce": False, "dtype": F32},
        # power iteration / PageRank on a graph, ten steps a pass
        {"name": "graph-21", "kind": "graph", "scale": 21, "edge_factor": 16, "iters": 10},
        # the two profiling matrices of the benchmark, a fifth of their size
        {"name": "medium-200000", "kind": "medium", "rows": 200_000, "cols": 1_000_000, "format": "K6", "dtype": F32},
        {"name": "long-9001", "kind": "long", "rows": 9_001, "cols": 1_000_000, "dtype": F32},
        # a web-like matrix, every strip of rows with the format that suits it
        {"name": "split-400000", "kind": "split", "rows": 400_000, "cap": 100_000, "dtype": F32},
        # a host program that calls the library for one product and keeps its own arrays
        {"name": "host-1024x1024", "kind": "host", "nx": 1024, "ny": 1024, "pipelined": False, "dtype": F64},
        # a matrix reassembled every step (Newton, time stepping): format and plan are made anew for one product
        {"name": "build-40000", "kind": "build", "nodes": 40_000, "blocks": 9, "format": "B1", "dtype": F64},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["rowgroup", "diag", "ell", "block", "sell", "powerlaw", "graph", "medium", "long", "split", "host", "build"])
    dtype = rng.choice([F32, F64])
    if kind == "rowgroup":
        return {"kind": kind, "rows": _log(rng, 300, 100_000), "mean": round(4.0 * 10.0 ** rng.random(), 1), "dtype": dtype}
    if kind in ("diag", "ell"):
        return {"kind": kind, "nx": _log(rng, 20, 2048), "ny": _log(rng, 20, 2048), "dtype": dtype}
    if kind in ("block", "sell"):
        return {"kind": kind, "nodes": _log(rng, 200, 65_000), "blocks": rng.randint(7, 27), "dtype": dtype}
    if kind == "powerlaw":
        return {"kind": kind, "rows": _log(rng, 2_000, 4_000_000), "tlb": rng.choice([4, 8, 16, 32, 3, 11]), "staged": rng.random() < 0.5,
                "warp_reduce": rng.random() < 0.3, "dtype": dtype}
    if kind == "graph":
        return {"kind": kind, "scale": rng.randint(11, 20), "edge_factor": rng.randint(4, 24), "iters": rng.randint(2, 12)}
    if kind == "medium":
        return {"kind": kind, "rows": _log(rng, 500, 200_000), "cols": _log(rng, 20_000, 1_000_000), "format": rng.choice(["K4", "K6", "K8"]), "dtype": dtype}
    if kind == "long":
        return {"kind": kind, "rows": _log(rng, 20, 7_000), "cols": _log(rng, 20_000, 1_000_000), "dtype": dtype}
    if kind == "split":
        return {"kind": kind, "rows": _log(rng, 5_000, 300_000), "cap": _log(rng, 5_000, 100_000), "dtype": dtype}
    if kind == "host":
        return {"kind": kind, "nx": _log(rng, 40, 1024), "ny": _log(rng, 40, 1024), "pipelined": rng.random() < 0.5, "dtype": dtype}
    return {"kind": kind, "nodes": _log(rng, 300, 30_000), "blocks": rng.randint(5, 9), "format": rng.choice(["B1", "K2", "K3", "K9"]), "dtype": dtype}


# ---- matrices, on the GPU ------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _torch_type(case):
    return torch.float64 if case.get("dtype") == F64 else torch.float32


def _uniform(g, n, dtype, lo=-1.0, hi=1.0):
    return torch.rand(n, generator=g, device="cuda", dtype=dtype) * (hi - lo) + lo


def _host_csr(n_rows, n_cols, lengths, cols, vals):
    indptr = torch.zeros(n_rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lengths, 0, out=indptr[1:])
    return CsrMatrix(n_rows, n_cols, indptr.cpu().numpy(), cols.to(torch.int32).cpu().numpy().view(np.uint32), vals.cpu().numpy())


def _random_columns(g, lengths, n_cols, dtype):
    """Rows of about the given lengths: uniformly random columns, sorted, duplicates of a row dropped."""
    n = lengths.shape[0]
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lengths)
    cols = torch.randint(0, n_cols, rows.shape, generator=g, device="cuda")
    key = torch.unique(rows * n_cols + cols)
    rows = torch.div(key, n_cols, rounding_mode="floor")
    return _host_csr(n, n_cols, torch.bincount(rows, minlength=n), key - rows * n_cols, _uniform(g, key.shape, dtype))


def _zipf(g, n, exponent, cap):
    k = torch.arange(1, cap + 1, dtype=torch.float64, device="cuda")
    cdf = torch.cumsum(k**-exponent, 0)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
    return torch.clamp(torch.searchsorted(cdf, u) + 1, max=cap)


def _zipf_mean(exponent, cap):
    k = np.arange(1, cap + 1, dtype=np.float64)
    p = k**-exponent
    return float((p * k).sum() / p.sum())


def _stencil(case, g):
    """-div(c grad u) on an nx x ny mesh with a random coefficient per cell face; rows are strictly diagonally dominant."""
    nx, ny, dt = case["nx"], case["ny"], _torch_type(case)
    n = nx * ny
    i = torch.arange(n, device="cuda")
    ix, iy = i % nx, torch.div(i, nx, rounding_mode="floor")
    east, north = _uniform(g, n, dt, 0.5, 1.5), _uniform(g, n, dt, 0.5, 1.5)
    west, south = torch.roll(east, 1), torch.roll(north, nx)
    cols = torch.stack([i - nx, i - 1, i, i + 1, i + nx], 1)
    vals = torch.stack([-south, -west, east + west + north + south, -east, -north], 1)
    keep = torch.stack([iy > 0, ix > 0, ix >= 0, ix < nx - 1, iy < ny - 1], 1)
    return _host_csr(n, n, keep.sum(1), cols[keep], vals[keep])


def _fem(case, g):
    """Dense 3 x 3 blocks: `blocks` distinct block columns a node inside a window of 8193 nodes (or of all), the diagonal one among them."""
    nb, k, dt = case["nodes"], case["blocks"], _torch_type(case)
    w = min(8193, nb)
    i = torch.arange(nb, device="cuda")
    start = torch.clamp(i - w // 2, 0, nb - w)
    off = torch.randint(0, w - k + 1, (nb, k - 1), generator=g, device="cuda").sort(1).values + torch.arange(k - 1, device="cuda")
    diag = (i - start)[:, None]
    bcol = torch.cat([off + (off >= diag), diag], 1).sort(1).values + start[:, None]
    cols = (bcol[:, :, None] * 3 + torch.arange(3, device="cuda")).reshape(nb, 1, 3 * k).expand(nb, 3, 3 * k).reshape(-1)
    vals = torch.randn(cols.shape, generator=g, device="cuda", dtype=dt)
    return _host_csr(3 * nb, 3 * nb, torch.full((3 * nb,), 3 * k, dtype=torch.int64, device="cuda"), cols, vals)


def _matrix(case, g):
    kind, dt = case["kind"], _torch_type(case)
    if kind == "rowgroup":
        mean = torch.full((case["rows"],), case["mean"], device="cuda")
        return _random_columns(g, torch.clamp(torch.poisson(mean, generator=g).to(torch.int64), min=1), case["rows"], dt)
    if kind in ("diag", "ell", "host"):
        return _stencil(case, g)
    if kind in ("block", "sell", "build"):
        return _fem(case, g)
    if kind == "powerlaw":
        return _random_columns(g, _zipf(g, case["rows"], 2.1, min(500_000, case["rows"])), case["rows"], dt)
    if kind == "medium":
        return _random_columns(g, torch.randint(40, 121, (case["rows"],), generator=g, device="cuda"), case["cols"], dt)
    if kind == "long":
        return _random_columns(g, torch.randint(1000, 3001, (case["rows"],), generator=g, device="cuda"), case["cols"], dt)
    return _random_columns(g, _zipf(g, case["rows"], 1.8, min(case["cap"], case["rows"])), case["rows"], dt)  # split


# ---- formats -------------------------------------------------------------------------------------------------------
def _graph(nodes, template, threads, reduce=1, dense="dense compress"):
    return {"dense": dense, "subs": [{"graph": template, "nodes": nodes, "template": template, "threads": threads, "row_reduce": reduce}]}


_FORMATS = {
    "K2": _graph(["row_padding 128 1", "blb_row_evenly 128", "tlb_row"], "K2", 256),
    "K3": _graph(["row_padding 32 1", "tlb_row"], "K3", 128),
    "K4": _graph(["wlb_col_fixed 64"], "K4", 256),
    "K6": _graph(["row_padding 32 1", "blb_row_evenly 32", "tlb_col_fixed 4"], "K6", 128, 4),
    "K8": _graph(["row_padding 4 1", "blb_row_evenly 4", "wlb_col_fixed 64"], "K8", 128, 4),
    "K9": _graph(["tlb_nnz 16"], "K9", 128, 2),
    "B1": _graph(["block_value 3 3"], "B1", 128),
    "D1": _graph(["diag_value 64"], "D1", 128),
}


def _format(case):
    kind = case["kind"]
    if kind == "rowgroup":
        return _graph(["row_padding 64 1", "blb_row_evenly 64", "tlb_col_fixed 4"], "K6", 128)
    if kind == "powerlaw":
        return _graph([f"tlb_nnz {case['tlb']}"], "K10" if case["warp_reduce"] else "K9", 128, 2 if case["staged"] else 1)
    if kind == "long":
        return _graph(["blb_col_fixed 1024"], "K7", 128)
    return _FORMATS[{"diag": "D1", "host": "D1", "ell": "K3", "block": "B1", "sell": "K2"}.get(kind) or case["format"]]


def _split(ctx, m):
    """Rows sorted by length and cut where it passes 128, 1024, 8192: SELL-like, row-grouped and long-row strips."""
    hm = Matrix.from_csr(m)
    cm = hm.dense("dense sort 1\ndense rowdiv_exp 128 4096 8\ndense compress")
    lines, launch = [], []
    for i in range(cm.n_subs):
        _, _, _, longest = cm.sub_rows(i)
        f = _FORMATS["K2"] if longest <= 128 else _FORMATS["K6"] if longest <= 1024 else _graph(["blb_col_fixed 1024"], "K7", 128)
        s = f["subs"][0]
        lines += [f"sub {i} {node}" for node in s["nodes"]] + [f"sub {i} template {s['template']}"]
        launch.append((s["threads"], s["row_reduce"]))
    fmt = cm.execute("\n".join(lines))
    group = fmt.upload(ctx)
    for i, (threads, reduce) in enumerate(launch):
        tuner.set_launch(fmt, group, i, threads, reduce)
    cm.close()
    hm.close()
    return fmt, group


_CONTEXT = None


def _context():
    """The one context that a program keeps per GPU."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = capi.Context(torch.cuda.current_device())
    return _CONTEXT


def prepare(case, seed):
    ctx, g, kind = _context(), _generator(seed), case["kind"]
    if kind == "graph":
        return _prepare_graph(ctx, case, seed)
    m = _matrix(case, g)
    x = _uniform(g, m.n_cols, _torch_type(case))
    s = {"kind": kind, "ctx": ctx}
    if kind == "build":
        return {**s, "m": m, "format": _format(case), "x": x, "y": torch.zeros(m.n_rows, dtype=x.dtype, device="cuda")}
    if kind == "host" and case["pipelined"]:
        # at most four pieces of rows, cut at multiples of 32
        chunks = tuner.build_row_chunks(ctx, m, _format(case), 4, align=32)
        return {**s, "chunks": [c[1:] for c in chunks], "keep": [c[0] for c in chunks], "x": x.cpu().pin_memory(),
                "y": torch.zeros(m.n_rows, dtype=x.dtype).pin_memory()}
    s["format"], s["group"] = _split(ctx, m) if kind == "split" else tuner.build(ctx, m, _format(case))
    if kind == "host":
        return {**s, "x": x.cpu().numpy()}
    return {**s, "x": x, "y": torch.zeros(m.n_rows, dtype=x.dtype, device="cuda")}


def _prepare_graph(ctx, case, seed):
    """The benchmark's loop on one GPU: vertices by column count, those with an empty row last, rows without non-zeros dropped."""
    scale, ef, n, dev = case["scale"], case["edge_factor"], 1 << case["scale"], torch.device("cuda")
    deg, cdeg = matrices_gpu.rmat_degrees(scale, ef, seed % 100_003, dev)
    labels, inverse = matrices_gpu.hotness_labels(cdeg, deg)
    active = int((deg > 0).sum().item())
    m = matrices_gpu.to_host_csr(*matrices_gpu.rmat_block(scale, ef, seed % 100_003, 0, active, dev, labels, inverse), n)
    m.values *= np.float32(1.0 / ef)  # keeps x in range however many steps are taken
    fmt, group = tuner.build(ctx, m, _graph(["tlb_nnz 32"], "K9", 128, dense="dense sort 1073741824 | dense compress"))
    bufs = [torch.zeros(n, device="cuda") for _ in range(2)]
    loop = capi.DistLoop(ctx, [(group, 0, active)], n)
    return {"kind": "graph", "format": fmt, "group": group, "loop": loop, "bufs": bufs, "x": matrices_gpu.rmat_x(scale, seed % 100_003, dev)[inverse].contiguous(),
            "iters": case["iters"]}


# ---- one pass ------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "graph":
        bufs = state["bufs"]
        return bufs[state["loop"].iterate(state["x"].data_ptr(), [b.data_ptr() for b in bufs], None, state["iters"])]
    if kind == "build":
        fmt, group = tuner.build(state["ctx"], state["m"], state["format"])
        group.spmv(state["x"].data_ptr(), state["y"].data_ptr(), "auto")
        state["ctx"].synchronize()
        group.close()
        fmt.close()
        return state["y"]
    if kind == "host":
        if "group" in state:
            return state["group"].spmv_host(state["x"])
        capi.spmv_host_pipelined(state["ctx"], state["chunks"], state["x"].data_ptr(), state["y"].data_ptr())
        return state["y"]
    # every row of these matrices has a non-zero, so y is cleared only where a kernel accumulates into it
    state["group"].spmv(state["x"].data_ptr(), state["y"].data_ptr(), "auto")
    return state["y"]


# ---- what a pass cannot do without, and how far results may be off -----------------------------------------------------
def work(case):
    """Bytes: the matrix once (a value and a 4-byte column per non-zero, a 4-byte offset per row; a column per block or an offset
    per diagonal where the format has those), x once, y once. Random
    matrices by their expected sizes, before duplicate columns of a row are dropped."""
    kind, sv = case["kind"], 8 if case.get("dtype") == F64 else 4
    per_nz = sv + 4.0
    passes = 1
    if kind == "graph":
        rows = cols = 1 << case["scale"]
        nnz, passes = rows * case["edge_factor"], case["iters"]
    elif kind == "rowgroup":
        rows = cols = case["rows"]
        nnz = rows * case["mean"]
    elif kind in ("diag", "ell", "host"):
        nx, ny = case["nx"], case["ny"]
        rows = cols = nx * ny
        nnz = 5 * rows - 2 * (nx + ny)
        per_nz = per_nz if kind == "ell" else sv
    elif kind in ("block", "sell", "build"):
        rows = cols = 3 * case["nodes"]
        nnz = 9 * case["nodes"] * case["blocks"]
        per_nz = sv + 4.0 / 9.0 if kind == "block" else per_nz
    elif kind == "powerlaw":
        rows = cols = case["rows"]
        nnz = rows * _zipf_mean(2.1, min(500_000, rows))
    elif kind == "split":
        rows = cols = case["rows"]
        nnz = rows * _zipf_mean(1.8, min(case["cap"], rows))
    else:
        rows, cols = case["rows"], case["cols"]
        nnz = rows * (80 if kind == "medium" else 2000)
    offsets = 0 if kind in ("diag", "host") else 4 * rows
    return {"bytes": passes * (nnz * per_nz + offsets + sv * (rows + cols)), "flops": passes * 2.0 * nnz}


def tolerance(case):
    # sums of 32- or 64-bit products in another order; `max` for the rows whose sum cancels
    if case.get("dtype") == F64:
        return {"rel": 1e-13, "max": 1e-11}
    return {"rel": 1e-5, "max": 1e-3}
