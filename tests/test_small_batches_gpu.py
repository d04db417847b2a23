"""Small batches are sorted, netted and cut into row units by one CTA in shared
memory (up to 2048 lines), which up to 512 lines also ends the batch; few
relocation copies stay with that CTA then, more go back to all of them;
batches up to 32768 lines run on one CTA per SM.  At each
of these edges the adjacency, the degree property, the colours and the
statistics must be the oracle's.

Oracle rules followed: HI/all_structure_undir.cuh:96-110,
HI/gpuFunctions_undir.cuh:118-142, HB/all_structure_undir.cuh:110-119."""
import numpy as np
import pytest

import dyncolor_b200 as dc
import pyoracle as po
from helpers import er_graph, oracle_graph, to_dc_changes

pytestmark = pytest.mark.gpu


def _lines(rng, n, k, a, b, p_del):
    """k lines: deletions of edges that were loaded, insertions, both for one
    pair, repeats, and a few lines with an inst value that is ignored (ids of
    those may be anything)."""
    i = rng.integers(0, len(a), k)
    x, y = rng.integers(0, n, k), rng.integers(0, n, k)
    old = rng.random(k) < 0.5
    x, y = np.where(old, a[i], x), np.where(old, b[i], y)
    y = np.where(x == y, (y + 1) % n, y)
    flip = rng.random(k) < 0.5
    x, y = np.where(flip, y, x), np.where(flip, x, y)
    inst = (rng.random(k) >= p_del).astype(np.int32)
    if k >= 8:
        x[k // 4:k // 2], y[k // 4:k // 2] = x[:k // 2 - k // 4], y[:k // 2 - k // 4]
        inst[-1], x[-1], y[-1] = 7, n + 5, -3
    return po.as_changes(x, y, inst)


@pytest.mark.parametrize("variant,ov", [(dc.HI, po.HI), (dc.HB, po.HB)])
@pytest.mark.parametrize("k", [0, 1, 2, 31, 511, 512, 513, 1024, 2047, 2048, 2049, 32768, 32769])
@pytest.mark.parametrize("kw", [{}, dict(cuda_graph=True), dict(grid_ctas=1)])
def test_batches_at_the_edges_of_the_small_path(variant, ov, k, kw):
    n, a, b = er_graph(5000, 12, seed=4)
    # one row longer than a row-scan unit
    hub = np.arange(1, 4500, dtype=np.int32)
    a, b = dc.dedup(n, np.concatenate([a, np.zeros_like(hub)]), np.concatenate([b, hub]))
    col = dc.greedy_color(n, a, b)
    ctx = dc.Context(variant=variant, **kw)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    rng = np.random.default_rng(k)
    for p_del in (0.5, 1.0, 0.0):
        ch = _lines(rng, n, k, a, b, p_del)
        rc, so = g.apply_batch(ch, ov, po.SNAPSHOT)
        sg = ctx.apply_batch(to_dc_changes(ch))
        assert rc == po.OK and np.array_equal(ctx.colors(), g.colors())
        # (the oracle's covered entries count a repeated insertion twice)
        assert (sg.iterations, sg.seed_targets, sg.frontier_total) == (
            so.iterations, so.seed_targets, so.frontier_total)
        for v in np.concatenate([[0], ch["node1"][:40]]):
            if 0 <= v < n:
                assert np.array_equal(ctx.neighbors(v), g.neighbors(v))
    assert np.array_equal(ctx.prop(), g.prop())
    ctx.close()


@pytest.mark.parametrize("rows", [60, 64, 65, 900])
def test_relocations_on_both_sides_of_the_line(rows):
    """Insertions that overflow `rows` tight rows: their copies stay with one
    CTA up to 64 units and use all of them above; the pool grows on the way."""
    n = 2000
    x = np.repeat(np.arange(rows), 2).astype(np.int32)
    y = (1000 + (np.arange(2 * rows) % 1000)).astype(np.int32)
    a, b = dc.dedup(n, np.arange(n - 1, dtype=np.int32), np.arange(1, n, dtype=np.int32))
    col = dc.greedy_color(n, a, b)
    ctx = dc.Context(variant=dc.HI, slack=1.01)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    relocated = 0
    for step in range(12):
        ch = po.as_changes(x, 1000 + (y - 1000 + 37 * step) % 1000, np.ones(len(x), np.int32))
        rc, so = g.apply_batch(ch, po.HI, po.SNAPSHOT)
        sg = ctx.apply_batch(to_dc_changes(ch))
        relocated += sg.rows_relocated
        assert np.array_equal(ctx.colors(), g.colors()) and sg.iterations == so.iterations
        for v in (0, 1, rows - 1, rows, 1000, 1037, 1999):
            assert np.array_equal(ctx.neighbors(v), g.neighbors(v))
    assert relocated > rows
    ctx.close()


@pytest.mark.parametrize("at", [0, 1000, 2047])
def test_an_invalid_line_leaves_the_graph_as_it_was(at):
    n, a, b = er_graph(3000, 8, seed=5)
    col = dc.greedy_color(n, a, b)
    ctx = dc.Context(variant=dc.HB)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    rng = np.random.default_rng(at)
    ch = _lines(rng, n, 2048, a, b, 0.5)
    bad = ch.copy()
    bad["inst"][at], bad["node1"][at], bad["node2"][at] = 1, n, 3
    with pytest.raises(dc.DcError) as e:
        ctx.apply_batch(to_dc_changes(bad))
    assert e.value.status == dc.E_INVAL
    assert np.array_equal(ctx.colors(), col)
    rc, so = g.apply_batch(ch, po.HB, po.SNAPSHOT)
    sg = ctx.apply_batch(to_dc_changes(ch))
    assert np.array_equal(ctx.colors(), g.colors()) and sg.iterations == so.iterations
    assert np.array_equal(ctx.prop(), g.prop())
    ctx.close()


@pytest.mark.parametrize("variant,ov", [(dc.HI, po.HI), (dc.HB, po.HB)])
@pytest.mark.parametrize("n", [64, 65, 66, 65536, 65537])
def test_graphs_at_the_edges_of_the_launch_rules(variant, ov, n):
    """No index where no row can be long enough (n <= heavy_min_live), and one
    CTA per SM for HI up to 65536 vertices."""
    hub = np.arange(1, min(n, 3000), dtype=np.int32)
    a, b = dc.uniform_pairs(n, 4 * n, seed=6)
    a, b = dc.dedup(n, np.concatenate([a, np.zeros_like(hub)]), np.concatenate([b, hub]))
    col = dc.greedy_color(n, a, b)
    ctx = dc.Context(variant=variant, heavy_min_live=64)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    rng = np.random.default_rng(n)
    for _ in range(3):
        ch = _lines(rng, n, max(30, n // 8), a, b, 0.5)
        rc, so = g.apply_batch(ch, ov, po.SNAPSHOT)
        sg = ctx.apply_batch(to_dc_changes(ch))
        assert rc == po.OK and np.array_equal(ctx.colors(), g.colors())
        assert (sg.iterations, sg.seed_targets, sg.frontier_total) == (
            so.iterations, so.seed_targets, so.frontier_total)
    ctx.close()
