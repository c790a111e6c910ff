"""GPU: a search times what will run. Trials are the templates' kernels, with their launch parameters; the column-tiled layout is a
candidate of its own, and the result says which of the two it found faster."""
import numpy as np
import pytest

import refdump
from alphasparse_b200 import matrices as M, tuner

pytestmark = pytest.mark.gpu


def test_trials_time_the_templates_kernels(asp_ctx):
    m, x = M.from_row_lengths(np.random.default_rng(2).integers(40, 121, size=120_000), 1_000_000, seed=2)
    lines = []
    fmt, group, trials, desc = tuner.search(asp_ctx, m, quick=True, warmup=2, reps=20, log=lines.append)
    assert desc["layout"] == "auto" and group.layout_bytes() > 0, desc  # scattered columns: the layout wins
    assert any("column-tiled layout" in l for l in lines)
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(group.spmv_host(x), y_ref, scale, np.float32, str(desc))
    group.close()
    fmt.close()
    seen = 0
    one = [t for t in trials if t.dense == "dense compress"]
    for name in sorted({t.name for t in one})[:6]:
        t = min((t for t in one if t.name == name), key=lambda t: t.ms)
        cand = next(c for c in tuner.compressed_candidates(40, 120, 80.0, False) if c.name == name)
        f, g = tuner.build(asp_ctx, m, {"dense": t.dense, "subs": [{"graph": name, "nodes": cand.nodes, "template": cand.template, "threads": t.launch[0], "row_reduce": t.launch[1]}]}, "none")
        own = g.time(3, 50)[0]
        assert 0.7 * own < t.ms < 1.5 * own, (name, t.ms, own)
        seen += 1
        g.close()
        f.close()
    assert seen >= 3


def test_a_matrix_without_the_layout(asp_ctx):
    m, x = M.laplacian_2d(512, seed=1, dtype=np.float32)
    fmt, group, trials, desc = tuner.search(asp_ctx, m, quick=True, warmup=1, reps=5)
    assert desc["layout"] == "none" and group.layout_bytes() == 0
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(group.spmv_host(x), y_ref, scale, np.float32, str(desc))
    group.close()
    fmt.close()


def test_trials_of_a_small_matrix(asp_ctx):
    """Kernels for whole rows are no trials: they take no launch parameters. What they are worth is timed once per format."""
    m, x = M.from_row_lengths(np.random.default_rng(2).integers(40, 121, size=2_000), 3_000, seed=2)
    lines = []
    fmt, group, trials, desc = tuner.search(asp_ctx, m, quick=True, warmup=2, reps=20, log=lines.append)
    assert desc["layout"] == "auto" and (group.whole_rows() or group.n > 1), desc
    rows = [l for l in lines if "by what replaces its kernel" in l]
    names = {t.name for t in trials if t.dense == "dense compress"}
    assert 0 < len(rows) and all(any(n in l for n in names) for l in rows)
    y_ref, scale = refdump.csr_ref(m, x)
    refdump.assert_y(group.spmv_host(x), y_ref, scale, np.float32, str(desc))
    group.close()
    fmt.close()
    for name in sorted(names):
        t = min((t for t in trials if t.dense == "dense compress" and t.name == name), key=lambda t: t.ms)
        cand = next(c for c in tuner.compressed_candidates(40, 120, 80.0, False) if c.name == name)
        f, g = tuner.build(asp_ctx, m, {"dense": t.dense, "subs": [{"graph": name, "nodes": cand.nodes, "template": cand.template, "threads": t.launch[0], "row_reduce": t.launch[1]}]}, "none")
        own = g.time(3, 50)[0]
        assert not g.whole_rows() and 0.6 * own < t.ms < 1.7 * own, (name, t.ms, own)
        g.close()
        f.close()


def test_the_callers_timer_decides_without_a_layout():
    m, _ = M.uniform_random(500, 8, seed=3)
    desc, _, _ = tuner.search_with_timer(m, lambda fmt, tb, th, rd: 1.0)
    assert desc["layout"] == "auto"
