"""The work a user of this framework has it do, as measured cases.

A case names a graph family and size, a variant of the algorithm, an update
batch and the entry point it goes through; every size below comes from the
benchmark's and the tests' configurations or is a generic one.  The graph is
resident (loaded and coloured once, as a program that keeps a colouring up
to date holds it), and one pass applies a batch of change lines, reads the
colours, applies the inverse batch (the deleted edges return, the inserted
ones go) and reads the colours again, so the graph is the same before every
pass and a pass can be repeated on the same state.  The colours are never
reset: like a running service, each batch starts from the colouring the last
one left.

Kinds:
  update   one graph, Context.apply_batch (lines in host memory) or
           Context.apply_batch_device (lines already in device memory)
  batched  many graphs in one launch sequence (BatchedContext, replayed from
           a captured CUDA graph)
  job      a whole run of the command: create, load, colour, one batch, read,
           check, close

Families:
  rmat     R-MAT a=.57 b=c=.19, self-loops and duplicates removed
  er       uniform random pairs
  cl       Chung-Lu power law with exponent 2.1 and hubs up to n/20
"""
import math

import numpy as np
import torch

import dyncolor_b200 as dc
from dyncolor_b200.batched import BatchedContext


def listed():
    return [
        # A handful of edges of a small graph change: launches, waits and
        # host calls are all there is.
        dict(name="hi_er_1k_l20", kind="update", variant="hi", family="er", n=1_000, deg=8.0, lines=20,
             ins=0.5, entry="host"),
        # The same for the priority variant, on an odd-sized skewed graph.
        dict(name="hb_rmat_3001_l101", kind="update", variant="hb", family="rmat", n=3_001, deg=16.0, lines=101,
             ins=0.5, entry="host"),
        # The small benchmark configuration: R-MAT scale 16, 10,000 deletions
        # and 10,000 uniform absent insertions.
        dict(name="hi_rmat16_l20k", kind="update", variant="hi", family="rmat", n=65_536, deg=32.0, lines=20_000,
             ins=0.5, entry="host", ends="uniform"),
        dict(name="hb_rmat16_l20k", kind="update", variant="hb", family="rmat", n=65_536, deg=32.0, lines=20_000,
             ins=0.5, entry="host", ends="uniform"),
        # A large sparse graph without hubs and a small batch (a road or mesh
        # like graph between two refreshes).
        dict(name="hi_er_1m_l5k", kind="update", variant="hi", family="er", n=1_000_003, deg=6.0, lines=5_000,
             ins=0.5, entry="device"),
        # R-MAT scale 20, 100,000-line batches: the middle of the range.
        dict(name="hi_rmat20_l100k", kind="update", variant="hi", family="rmat", n=1 << 20, deg=32.0,
             lines=100_000, ins=0.5, entry="host"),
        # The priority variant on a large graph (R-MAT scale 22).
        dict(name="hb_rmat22_l250k", kind="update", variant="hb", family="rmat", n=1 << 22, deg=32.0,
             lines=250_000, ins=0.5, entry="device"),
        # The skewed-degree configuration, both variants: hub rows, masks of
        # several words, mostly insertions with one endpoint drawn by degree.
        dict(name="hi_cl_1m_l250k", kind="update", variant="hi", family="cl", n=1_000_000, deg=24.0,
             lines=250_000, ins=0.7, entry="host"),
        dict(name="hb_cl_1m_l250k", kind="update", variant="hb", family="cl", n=1_000_000, deg=24.0,
             lines=250_000, ins=0.7, entry="host"),
        # The benchmark's default workload: R-MAT scale 24, 1,000,000 lines.
        dict(name="hi_rmat24_l1m", kind="update", variant="hi", family="rmat", n=1 << 24, deg=32.0,
             lines=1_000_000, ins=0.5, entry="device"),
        # Many graphs of uneven size, each with its own batch, in one launch.
        dict(name="batched_hi_96", kind="batched", variant="hi", graphs=96, nmin=1_000, nmax=100_000,
             kmin=100, kmax=20_000),
        # One run of the command on a graph file's edges: everything is new.
        dict(name="job_hb_rmat18_l20k", kind="job", variant="hb", family="rmat", n=1 << 18, deg=32.0, lines=20_000,
             ins=0.5),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update"] * 8 + ["batched", "job"])
    variant = rng.choice(["hi", "hb"])
    if kind == "batched":
        return dict(kind=kind, variant=variant, graphs=rng.randint(16, 96), nmin=1_000,
                    nmax=_log_uniform(rng, 10_000, 100_000), kmin=100, kmax=_log_uniform(rng, 1_000, 20_000))
    family = rng.choice(["rmat", "rmat", "er", "cl"])
    n = _log_uniform(rng, 1_000, 300_000 if kind == "job" else 2_000_000 if variant == "hb" else 4_000_000)
    case = dict(kind=kind, variant=variant, family=family, n=n, deg=round(rng.uniform(4.0, 32.0), 2),
                lines=_log_uniform(rng, 10, max(20, n // 4)), ins=rng.choice([0.3, 0.5, 0.7]))
    if kind == "update":
        case["entry"] = rng.choice(["host", "device"])
        if family == "rmat":
            case["ends"] = rng.choice(["same", "uniform"])
    return case


# ---------------------------------------------------------------------------
# seeded graphs and batches, on the GPU
# ---------------------------------------------------------------------------

def _rmat_ends(g, n, m):
    scale = max(1, (n - 1).bit_length())
    u = torch.zeros(m, dtype=torch.int32, device="cuda")
    v = torch.zeros(m, dtype=torch.int32, device="cuda")
    for level in range(scale):
        r = torch.rand(m, generator=g, device="cuda")
        bu = r >= 0.76
        bv = ((r >= 0.57) & (r < 0.76)) | (r >= 0.95)
        u = (u << 1) | bu
        v = (v << 1) | bv
        del r, bu, bv
    return u, v


def _cl_cdf(n, deg):
    """Cumulative weights of a power law of exponent 2.1, largest n/20 of the
    average total."""
    w = (torch.arange(n, dtype=torch.float64, device="cuda") + 1.0) ** (-1.0 / 1.1)
    w *= deg * n / w.sum()
    w.clamp_(max=n / 20.0)
    c = torch.cumsum(w, 0)
    return c / c[-1]


def _cl_ends(g, cdf, m):
    r = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
    return torch.searchsorted(cdf, r).clamp_(max=len(cdf) - 1).int()


def _uniform_ends(g, n, m):
    return torch.randint(0, n, (m,), generator=g, device="cuda", dtype=torch.int32)


def _keys(n, u, v):
    """Distinct undirected pairs as sorted 64-bit keys."""
    lo, hi = torch.minimum(u, v), torch.maximum(u, v)
    keep = (lo != hi) & (hi < n)
    lo, hi = lo[keep].long(), hi[keep].long()
    return torch.unique((lo << 32) | hi)


def _graph(g, family, n, deg):
    m = max(1, int(n * deg / 2))
    cdf = None
    if family == "rmat":
        u, v = _rmat_ends(g, n, m)
    elif family == "cl":
        cdf = _cl_cdf(n, deg)
        u, v = _cl_ends(g, cdf, m), _cl_ends(g, cdf, m)
    else:
        u, v = _uniform_ends(g, n, m), _uniform_ends(g, n, m)
    return _keys(n, u, v), cdf


def _batch(g, keys, n, lines, ins, ends, cdf):
    """Change lines (k, 3) int32: deletions of distinct existing edges and
    insertions of distinct absent pairs, shuffled."""
    kd = min(lines - int(lines * ins), len(keys) // 2)
    ki = lines - kd
    pick = torch.unique(torch.randint(0, len(keys), (2 * kd + 16,), generator=g, device="cuda"))
    dele = keys[pick[torch.randperm(len(pick), generator=g, device="cuda")[:kd]]]
    more = 4 * ki + 64
    if ends == "rmat":
        u, v = _rmat_ends(g, n, more)
    elif ends == "degree":
        u, v = _cl_ends(g, cdf, more), _uniform_ends(g, n, more)
    else:
        u, v = _uniform_ends(g, n, more), _uniform_ends(g, n, more)
    new = _keys(n, u, v)
    at = torch.searchsorted(keys, new).clamp_(max=len(keys) - 1)
    new = new[keys[at] != new]
    new = new[torch.randperm(len(new), generator=g, device="cuda")[:ki]]
    key = torch.cat([dele, new])
    inst = torch.cat([torch.zeros(len(dele), dtype=torch.int32, device="cuda"),
                      torch.ones(len(new), dtype=torch.int32, device="cuda")])
    flip = torch.rand(len(key), generator=g, device="cuda") < 0.5
    lo, hi = (key >> 32).int(), (key & 0xFFFFFFFF).int()
    out = torch.stack([torch.where(flip, lo, hi), torch.where(flip, hi, lo), inst], 1)
    return out[torch.randperm(len(out), generator=g, device="cuda")].contiguous()


def _inverse(lines):
    out = lines.clone()
    out[:, 2] = 1 - out[:, 2]
    return out


def _host(lines):
    return lines.cpu().numpy().view(dc.CHANGE_DTYPE).reshape(-1).copy()


def _pairs(keys):
    return (keys >> 32).int().cpu().numpy(), (keys & 0xFFFFFFFF).int().cpu().numpy()


def _ends_of(case):
    if case["family"] == "cl":
        return "degree"
    if case["family"] == "rmat" and case.get("ends", "same") == "same":
        return "rmat"
    return "uniform"


def _pinned(n):
    return torch.empty(n, dtype=torch.int32).pin_memory().numpy()


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    variant = dc.HB if case["variant"] == "hb" else dc.HI
    order = dc.ORDER_LDF if variant == dc.HB else dc.ORDER_ID
    if case["kind"] == "batched":
        G = case["graphs"]
        rng = np.random.default_rng(G)  # sizes belong to the case, edges and lines to the seed
        ns = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), G)).astype(np.int64)
        degs = rng.uniform(8.0, 32.0, G)
        ks = np.exp(rng.uniform(math.log(case["kmin"]), math.log(case["kmax"]), G)).astype(np.int64)
        graphs, there, back = [], [], []
        for i in range(G):
            n = int(ns[i])
            keys, _ = _graph(g, "rmat" if i % 2 == 0 else "er", n, float(degs[i]))
            graphs.append((n, *_pairs(keys)))
            lines = _batch(g, keys, n, int(ks[i]), 0.5, "uniform", None)
            there.append(_host(lines))
            back.append(_host(_inverse(lines)))
        bc = BatchedContext(variant=variant, cuda_graph=True)
        bc.load(graphs)
        bc.ctx.init_colors(order)
        return dict(kind="batched", bc=bc, there=there, back=back, out=[_pinned(bc.n), _pinned(bc.n)])
    n = case["n"]
    keys, cdf = _graph(g, case["family"], n, case["deg"])
    lines = _batch(g, keys, n, case["lines"], case["ins"], _ends_of(case), cdf)
    a, b = _pairs(keys)
    del keys, cdf
    if case["kind"] == "job":
        return dict(kind="job", variant=variant, order=order, n=n, a=a, b=b, lines=_host(lines))
    ctx = dc.Context(variant=variant)
    ctx.load_edges(n, a, b)
    ctx.init_colors(order)
    there, back = lines, _inverse(lines)
    if case["entry"] == "host":
        there, back = _host(there), _host(back)
    torch.cuda.synchronize()
    return dict(kind="update", ctx=ctx, entry=case["entry"], there=there, back=back, out=[_pinned(n), _pinned(n)])


def _steps(st):
    return [st.iterations, st.seed_targets, st.frontier_total, st.slots_scanned, st.edges_inserted,
            st.edges_deleted, st.max_color]


def run(state):
    if state["kind"] == "job":
        ctx = dc.Context(variant=state["variant"])
        ctx.load_edges(state["n"], state["a"], state["b"])
        ctx.init_colors(state["order"])
        st = ctx.apply_batch(state["lines"])
        colors, bad = ctx.colors(), ctx.validate()
        ctx.close()
        return [colors, bad, _steps(st)]
    if state["kind"] == "batched":
        bc, res = state["bc"], []
        for lines, out in zip((state["there"], state["back"]), state["out"]):
            st = bc.apply(lines)
            res += [bc.ctx.colors(out), bc.iterations(), _steps(st)]
        return res
    ctx, res = state["ctx"], []
    for lines, out in zip((state["there"], state["back"]), state["out"]):
        if state["entry"] == "host":
            st = ctx.apply_batch(lines)
        else:
            st = ctx.apply_batch_device(lines.data_ptr(), len(lines))
        res += [ctx.colors(out), _steps(st)]
    return res


def work(case):
    """Lines read, the two rows of every line (ids and neighbour colours, at
    the average degree) read and its two slots written, colours written; the
    cascade behind a batch depends on the colouring and is not counted."""
    if case["kind"] == "batched":
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        n = case["graphs"] * (case["nmax"] - case["nmin"]) / max(hi - lo, 1e-9)
        lo, hi = math.log(case["kmin"]), math.log(case["kmax"])
        lines = case["graphs"] * (case["kmax"] - case["kmin"]) / max(hi - lo, 1e-9)
        deg, passes = 20.0, 2
    else:
        n, lines, deg = case["n"], case["lines"], case["deg"]
        passes = 1 if case["kind"] == "job" else 2
    per_line = 12 + 2 * (8 * deg + 4)
    total = passes * (lines * per_line + 4 * n)
    if case["kind"] == "job":
        total += 2 * 4 * n * deg + 12 * n  # the edge list read, the rows written and read, colours and check
    return {"bytes": float(total), "flops": 0.0}
