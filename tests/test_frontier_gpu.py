"""The recolouring loop finds each frontier from the last one (new and changed
vertices push their marks, members look for a witness, long searches are cut
into pieces) and computes a mex only where it can have changed.  Colours,
iterations, frontier sizes and covered entries must stay the oracle's on
graphs whose hub rows end at the edges of the pieces the loop cuts rows into:
a class-A row (32 slots), one round of a warp (128), a work unit (512), the
inline part of a search (512) plus a unit, and several units.

Oracle rules followed: HI/gpuFunctions_undir.cuh:229-284,
HB/gpuFunctions_undir.cuh:259-314."""
import numpy as np
import pytest

import dyncolor_b200 as dc
import pyoracle as po
from helpers import oracle_graph, to_dc_changes

pytestmark = pytest.mark.gpu

EDGES = (31, 32, 33, 127, 128, 129, 511, 512, 513, 640, 1023, 1024, 1025, 2500)


def _hubs(leaves, seed):
    """Hub i (the first vertices) has EDGES[i] neighbours among the leaves;
    the leaves carry a sparse random graph, so that cascades reach the hubs
    through low colours and back."""
    rng = np.random.default_rng(seed)
    h = len(EDGES)
    n = h + leaves
    a = np.concatenate([np.full(d, i) for i, d in enumerate(EDGES)] + [rng.integers(h, n, 2 * leaves)])
    b = np.concatenate([h + rng.permutation(leaves)[:d] for d in EDGES] + [rng.integers(h, n, 2 * leaves)])
    keep = a != b
    return (n, *dc.dedup(n, a[keep].astype(np.int32), b[keep].astype(np.int32)))


@pytest.mark.parametrize("variant,ov", [(dc.HI, po.HI), (dc.HB, po.HB)])
@pytest.mark.parametrize("kw", [dict(heavy_min_live=-1), dict(heavy_min_live=64), dict(unit_slots=128),
                                dict(grid_ctas=1), dict(cuda_graph=True)])
def test_rows_at_the_edges_of_the_loops_pieces(variant, ov, kw):
    n, a, b = _hubs(3000, seed=1)
    col = dc.greedy_color(n, a, b)
    ctx = dc.Context(variant=variant, **kw)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    es = dc.EdgeSet(n, a, b)
    for i in range(6):
        # small batches too: a handful of vertices and one with every hub in it
        k = (4, 60, 1500)[i % 3]
        ch = es.sample_batch(k // 2, k - k // 2, mode=dc.INS_DEGREE, seed=20 + i)
        rc, so = g.apply_batch(ch, ov, po.SNAPSHOT)
        sg = ctx.apply_batch(to_dc_changes(ch))
        assert rc == po.OK
        assert np.array_equal(ctx.colors(), g.colors())
        assert (sg.iterations, sg.seed_targets, sg.frontier_total, sg.slots_scanned) == (
            so.iterations, so.seed_targets, so.frontier_total, so.slots_scanned)
    assert ctx.validate() == 0
    ctx.close()


@pytest.mark.parametrize("variant,ov", [(dc.HI, po.HI), (dc.HB, po.HB)])
def test_improper_start_and_repeated_batches(variant, ov):
    """Colours that are not a greedy colouring (equal ends, gaps): no mex is
    known when the loop starts, and conflicts between members decide who
    stays."""
    rng = np.random.default_rng(3)
    n, a, b = _hubs(2600, seed=2)
    col = rng.integers(0, 9, n).astype(np.int32)
    ctx = dc.Context(variant=variant)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    for i in range(4):
        x, y = rng.integers(0, n, 400), rng.integers(0, n, 400)
        keep = x != y
        ch = po.as_changes(x[keep], y[keep], rng.integers(0, 2, keep.sum()))
        rc, so = g.apply_batch(ch, ov, po.SNAPSHOT, iter_cap=5000)
        sg = ctx.apply_batch(to_dc_changes(ch))
        assert rc == po.OK and np.array_equal(ctx.colors(), g.colors())
        assert (sg.iterations, sg.seed_targets, sg.frontier_total) == (
            so.iterations, so.seed_targets, so.frontier_total)
    ctx.close()


@pytest.mark.parametrize("variant,ov", [(dc.HI, po.HI), (dc.HB, po.HB)])
@pytest.mark.parametrize("clique", [250, 255, 256, 257, 300])
def test_colours_past_one_byte_in_indexed_rows(variant, ov, clique):
    """A clique with as many colours as vertices, hung with leaves so that its
    rows are indexed and reach behind it: walks of indexed rows that keep one
    byte per colour must still tell colours above it apart."""
    rng = np.random.default_rng(clique)
    n = clique + 1500
    x, y = np.triu_indices(clique, 1)
    lx, ly = rng.integers(0, clique, 12000), rng.integers(clique, n, 12000)
    a = np.concatenate([x, lx, clique + np.arange(1499)]).astype(np.int32)
    b = np.concatenate([y, ly, clique + 1 + np.arange(1499)]).astype(np.int32)
    a, b = dc.dedup(n, a, b)
    col = dc.greedy_color(n, a, b)
    assert col.max() >= clique - 1
    ctx = dc.Context(variant=variant, heavy_min_live=64)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    for i in range(5):
        # edges inside the clique go and come back, and some of the leaves'
        p, q = rng.integers(0, clique, 200), rng.integers(0, clique, 200)
        r, s = rng.integers(0, clique, 200), rng.integers(clique, n, 200)
        u, v = np.concatenate([p, r]), np.concatenate([q, s])
        keep = u != v
        ch = po.as_changes(u[keep], v[keep], rng.integers(0, 2, keep.sum()))
        rc, so = g.apply_batch(ch, ov, po.SNAPSHOT)
        sg = ctx.apply_batch(to_dc_changes(ch))
        assert rc == po.OK and np.array_equal(ctx.colors(), g.colors())
        assert (sg.iterations, sg.seed_targets, sg.frontier_total) == (
            so.iterations, so.seed_targets, so.frontier_total)
    ctx.close()


@pytest.mark.parametrize("variant,ov", [(dc.HI, po.HI), (dc.HB, po.HB)])
@pytest.mark.parametrize("degree", [32, 34, 40])
def test_every_row_just_past_the_short_search(variant, ov, degree):
    """A ring lattice whose rows all end just past the length up to which
    witness searches run 32 rows at a time, with a first frontier of nearly
    every vertex: each search that goes on takes a region of its own."""
    rng = np.random.default_rng(degree)
    n = 20000
    v = np.arange(n, dtype=np.int32)
    a = np.concatenate([v] * (degree // 2))
    b = np.concatenate([(v + k + 1) % n for k in range(degree // 2)]).astype(np.int32)
    a, b = dc.dedup(n, a, b)
    col = rng.integers(0, degree, n).astype(np.int32)
    ctx = dc.Context(variant=variant, slack=1.01)
    ctx.load_edges(n, a, b)
    ctx.set_colors(col)
    g = oracle_graph(n, a, b, col)
    for i in range(2):
        x = rng.integers(0, n, 30000)
        y = (x + 1 + rng.integers(0, degree // 2, 30000)) % n
        ch = po.as_changes(x, y, rng.integers(0, 2, 30000))
        rc, so = g.apply_batch(ch, ov, po.SNAPSHOT)
        sg = ctx.apply_batch(to_dc_changes(ch))
        assert rc == po.OK and np.array_equal(ctx.colors(), g.colors())
        assert (sg.iterations, sg.seed_targets, sg.frontier_total) == (
            so.iterations, so.seed_targets, so.frontier_total)
    ctx.close()


@pytest.mark.parametrize("order", [dc.ORDER_ID, dc.ORDER_LDF])
@pytest.mark.parametrize("kw", [{}, dict(unit_slots=128), dict(grid_ctas=1)])
def test_initial_colouring_of_rows_at_the_edges_of_its_units(order, kw):
    n, a, b = _hubs(3000, seed=5)
    deg = np.bincount(np.concatenate([a, b]), minlength=n)
    seq = np.arange(n) if order == dc.ORDER_ID else np.lexsort((np.arange(n), -deg))
    ctx = dc.Context(variant=dc.HB, **kw)
    ctx.load_edges(n, a, b)
    g = oracle_graph(n, a, b, np.zeros(n, np.int32))
    for _ in range(2):
        ctx.init_colors(order)
        g.greedy_in_order(seq.astype(np.int32))
        assert np.array_equal(ctx.colors(), g.colors())
    ctx.close()
