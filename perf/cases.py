"""The calls whose speed users of the framework feel, as a list of cases.

A case names a graph family and its size, the edge weights, how many queries
of each kind run over it, and the entry point they go through.  The families
and parameters are the ones the generators and the benchmark provide: R-MAT
(edge factor 16, .57/.19/.19), the 4-neighbour grid with 10% of its edges
deleted and 0.1% shortcuts, Chung-Lu with exponent 2.1, and a directed graph
from an edge list.  Graph, weights and sources all come from the seed.
"""
import math

import numpy as np
import torch

import cgp_b200 as cgp

KINDS = ("bfs", "sssp", "khop", "wcc")

# Keys that a case may leave out.
DEFAULTS = {
    "weights": "none",      # none | u32 (uniform [1, 64]) | f32 (uniform [1, 100)) | lognormal (f32)
    "bfs": 0, "sssp": 0, "khop": 0, "wcc": 0,
    "entry": "batch",       # batch (device output) | host (numpy result) | replenish (slot reuse)
    "layout": "vertex",     # vertex: [V][Q], query: [Q][V]
    "mode": "hybrid",       # RunOptions.traversal_mode
    "offsets64": False,
    "slots": 64,            # replenish only
}


def listed():
    return [
        # one request on a small graph: nothing but latency
        dict(name="point_bfs_rmat12", graph="rmat", scale=12, bfs=1),
        # a few routes on a small road-like graph: hundreds of levels, each tiny
        dict(name="routes_grid96_q16", graph="grid", rows=96, cols=97, weights="f32", sssp=16),
        # the small benchmark workload: one mask word of BFS over R-MAT 16
        dict(name="bfs_rmat16_q64", graph="rmat", scale=16, bfs=64),
        # the flagship step's two halves (256 BFS, then 256 SSSP) at a scale whose
        # values exceed L2 many times
        dict(name="bfs_rmat20_q256", graph="rmat", scale=20, bfs=256),
        dict(name="sssp_rmat20_q256", graph="rmat", scale=20, weights="u32", sssp=256),
        # deep traversal of a wide group on a road-like graph
        dict(name="sssp_grid700x900_q1024", graph="grid", rows=700, cols=900, weights="f32",
             sssp=1024),
        # a heterogeneous batch as in the reference's hybrid engine: all four kinds at once
        dict(name="mixed_rmat17_q48", graph="rmat", scale=17, weights="u32", bfs=24, sssp=16,
             khop=6, wcc=2, layout="query"),
        # power-law graph, log-normal weights, large batch split by kind, odd sizes
        dict(name="mixed_chunglu300k_q1000", graph="chung_lu", vertices=300007,
             weights="lognormal", bfs=501, sssp=499),
        # directed graph with 64-bit offsets: gathers go over the transpose
        dict(name="sssp_directed200k_q100", graph="directed", vertices=200003, degree=12,
             weights="u32", sssp=100, offsets64=True),
        # neighbourhood queries whose result the caller wants as a numpy array
        dict(name="khop_rmat18_q90_host", graph="rmat", scale=18, khop=90, entry="host"),
        # components of a large road-like graph
        dict(name="wcc_grid1100x1300", graph="grid", rows=1100, cols=1300, wcc=1),
        # a stream of mixed requests through reused bitmask slots
        dict(name="replenish_rmat15_q300", graph="rmat", scale=15, weights="u32", bfs=180,
             sssp=90, khop=30, entry="replenish", slots=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    shape = rng.choice(["bfs", "bfs", "sssp", "sssp", "grid", "mixed", "chung_lu", "directed",
                        "host", "wcc", "replenish"])
    c = {"mode": rng.choice(["hybrid"] * 8 + ["push", "pull"])}
    if shape in ("bfs", "sssp"):
        c.update(graph="rmat", scale=rng.randint(10, 19))
        c[shape] = _log_int(rng, 1, 400)
        if shape == "sssp":
            c["weights"] = rng.choice(["u32", "u32", "f32", "none"])
        c["offsets64"] = rng.random() < 0.2
        c["layout"] = rng.choice(["vertex", "vertex", "query"])
    elif shape == "grid":
        c.update(graph="grid", rows=_log_int(rng, 40, 600), cols=_log_int(rng, 40, 600),
                 weights=rng.choice(["f32", "u32"]), sssp=_log_int(rng, 1, 700), mode="hybrid")
    elif shape == "mixed":
        c.update(graph="rmat", scale=rng.randint(12, 17), weights=rng.choice(["u32", "f32"]),
                 bfs=rng.randint(1, 60), sssp=rng.randint(1, 60), khop=rng.randint(0, 20),
                 wcc=rng.randint(0, 2), layout=rng.choice(["vertex", "query"]))
    elif shape == "chung_lu":
        c.update(graph="chung_lu", vertices=_log_int(rng, 5000, 200000), weights="lognormal",
                 bfs=_log_int(rng, 10, 500), sssp=_log_int(rng, 10, 500))
    elif shape == "directed":
        c.update(graph="directed", vertices=_log_int(rng, 2000, 200000),
                 degree=rng.randint(2, 16), weights=rng.choice(["u32", "none"]),
                 bfs=rng.randint(0, 100), sssp=rng.randint(1, 150),
                 offsets64=rng.random() < 0.5)
    elif shape == "host":
        c.update(graph="rmat", scale=rng.randint(12, 18), entry="host")
        c[rng.choice(["khop", "bfs"])] = rng.randint(3, 100)
    elif shape == "wcc":
        c.update(graph=rng.choice(["rmat", "grid"]), wcc=1)
        if c["graph"] == "rmat":
            c["scale"] = rng.randint(12, 19)
        else:
            c.update(rows=_log_int(rng, 100, 900), cols=_log_int(rng, 100, 900))
    else:
        n = _log_int(rng, 20, 300)
        c.update(graph="rmat", scale=rng.randint(10, 15), weights="u32", entry="replenish",
                 bfs=n - n // 3, sssp=n // 3, khop=rng.randint(0, 20),
                 slots=rng.choice([32, 64, 128]), mode="hybrid")
    return c


# ------------------------------------------------------------------- inputs
def _full(case):
    return {**DEFAULTS, **case}


def _host_graph(c, seed):
    if c["graph"] == "rmat":
        g = cgp.gen_rmat(c["scale"], 16, 0.57, 0.19, 0.19, seed=seed)
    elif c["graph"] == "grid":
        g = cgp.gen_grid(c["rows"], c["cols"], 0.1, 0.001, seed=seed)
    elif c["graph"] == "chung_lu":
        g = cgp.gen_chung_lu(c["vertices"], 2.1, 16.0, seed=seed)
    else:
        # directed: uniform sources, destinations skewed towards low ids
        r = np.random.default_rng(seed)
        n, m = c["vertices"], c["vertices"] * c["degree"]
        dst = (n * r.random(m) ** 2).astype(np.int64)
        g = cgp.csr_from_edges(n, r.integers(0, n, m), np.minimum(dst, n - 1), symmetrize=False)
    if c["weights"] == "u32":
        g = g.with_weights("u32", 1, 64, seed=seed + 1)
    elif c["weights"] == "f32":
        g = g.with_weights("f32", 1.0, 100.0, seed=seed + 1)
    elif c["weights"] == "lognormal":
        g = g.with_weights("f32", 0.0, 1.0, seed=seed + 1, lognormal=True)
    return g


def _sources(c, g, n, seed):
    """Half from a corner (grid) or the top 1% of hubs (Chung-Lu), the rest
    uniform among vertices with out-edges."""
    V = g.num_vertices
    near = None
    if c["graph"] == "grid":
        r, k = np.divmod(np.arange(V), c["cols"])
        near = (r < max(2, c["rows"] // 10)) & (k < max(2, c["cols"] // 10))
        near &= g.degrees() > 0
    elif c["graph"] == "chung_lu":
        near = np.zeros(V, bool)
        near[np.argsort(-g.degrees(), kind="stable")[: max(1, V // 100)]] = True
    if near is None or n < 2 or not near.any():
        return g.pick_sources(n, seed=seed)
    a = g.pick_sources(n // 2, seed=seed, allowed=near.astype(np.uint8))
    return np.concatenate([a, g.pick_sources(n - n // 2, seed=seed + 1)])


def _inputs(case, seed):
    c = _full(case)
    base = 1 + 16 * int(seed)
    g = _host_graph(c, base)
    rng = np.random.default_rng(base)
    queries = []
    for i, kind in enumerate(KINDS):
        if not c[kind]:
            continue
        src = [0] * c[kind] if kind == "wcc" else _sources(c, g, c[kind], base + 2 + 2 * i)
        for s in src:
            k = int(rng.integers(2, 7)) if kind == "khop" else 0
            queries.append(cgp.QueryDescriptor(int(s), kind, k))
    if c["entry"] == "replenish":  # requests arrive in mixed order
        queries = [queries[i] for i in rng.permutation(len(queries))]
    return c, g, queries


def prepare(case, seed):
    c, g, queries = _inputs(case, seed)
    graph = cgp.CsrGraph(g, offsets64=c["offsets64"],
                         symmetric=None if c["graph"] == "directed" else True)
    st = {"case": c, "graph": graph, "queries": queries}
    if c["entry"] == "batch":
        n = len(queries)
        shape = (n, g.num_vertices) if c["layout"] == "query" else (g.num_vertices, n)
        st["out"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    st["options"] = cgp.RunOptions(traversal_mode=c["mode"],
                                   enable_replenishment=c["entry"] == "replenish")
    return st


# ---------------------------------------------------------------------- run
def _by_kind(c, words):
    """The result's 4-byte words per query kind: depths, labels and integer
    distances as int32, distances over float weights as float32."""
    axis = 0 if c["layout"] == "query" else 1
    out, at = {}, 0
    for kind in KINDS:
        if c[kind]:
            part = words[at:at + c[kind]] if axis == 0 else words[:, at:at + c[kind]]
            if kind == "sssp" and c["weights"] in ("f32", "lognormal"):
                part = part.view(torch.float32)
            out[kind] = part
            at += c[kind]
    return out


def run(st):
    c = st["case"]
    if c["entry"] == "replenish":
        r = cgp.run_replenish_pipeline(st["graph"], st["queries"], options=st["options"],
                                       slots=c["slots"])
        return r.values.view(np.int32)
    batch = cgp.HybridQueryBatch(st["queries"])
    if c["entry"] == "host":
        r = cgp.run_heterogeneous(st["graph"], batch, options=st["options"], layout=c["layout"])
        return r.values.view(np.int32)
    cgp.run_heterogeneous(st["graph"], batch, options=st["options"], layout=c["layout"],
                          out=st["out"])
    return _by_kind(c, st["out"])


# --------------------------------------------------------------- accounting
def _sizes(c):
    if c["graph"] == "rmat":
        v = 1 << c["scale"]
        # share of the 2 x 16 V entries left after removing loops and duplicates
        return v, int(2 * 16 * v * min(0.96, 0.62 + 0.0155 * c["scale"]))
    if c["graph"] == "grid":
        v = c["rows"] * c["cols"]
        return v, int(2 * 2 * v * 0.9)
    if c["graph"] == "chung_lu":
        return c["vertices"], int(0.8 * 16 * c["vertices"])
    return c["vertices"], c["vertices"] * c["degree"]


def work(case):
    """The CSR (offsets, columns, weights if a query uses them) read once, the
    [V][Q] result written once."""
    c = _full(case)
    v, e = _sizes(c)
    n = sum(c[k] for k in KINDS)
    per_edge = 4 + (4 if c["sssp"] and c["weights"] != "none" else 0)
    return {"bytes": e * per_edge + (v + 1) * (8 if c["offsets64"] else 4) + 4 * v * n, "flops": 0}


# -------------------------------------------------------------------- exact
def _bellman_ford(row, col, w, sources, V):
    """float64 distances [V][n] over in-edges (row/col/w list each vertex's)."""
    d = torch.full((V, len(sources)), math.inf, dtype=torch.float64, device=row.device)
    q = torch.arange(len(sources), device=row.device)
    d[torch.as_tensor(np.asarray(sources), device=row.device).long(), q] = 0.0
    while True:
        cand = d[col] + w.unsqueeze(1)
        new = torch.minimum(d, torch.segment_reduce(cand, "min", offsets=row, axis=0,
                                                    initial=math.inf))
        if torch.equal(new, d):
            return d
        d = new


def exact(case, seed):
    """SSSP distances over float weights in 64 bits; the other results are
    whole numbers."""
    c = _full(case)
    if not c["sssp"] or c["weights"] not in ("f32", "lognormal") or c["entry"] != "batch":
        return None
    v, e = _sizes(c)
    rounds = 2.5 * (c["rows"] + c["cols"]) if c["graph"] == "grid" else 40
    if rounds * e * c["sssp"] > 6e11:
        return None
    c, g, queries = _inputs(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    row = torch.from_numpy(np.asarray(g.row_offsets, np.int64)).to(dev)
    col = torch.from_numpy(g.col_indices).to(dev).long()
    w = torch.from_numpy(g.weights).to(dev).double()
    src = [x.source for x in queries if x.kind == "sssp"]
    step = max(1, int(4e8 // max(1, g.num_edges)))
    d = torch.cat([_bellman_ford(row, col, w, src[i:i + step], g.num_vertices)
                   for i in range(0, len(src), step)], dim=1)
    d = d.t() if c["layout"] == "query" else d
    return {k: (d if k == "sssp" else None) for k in KINDS if c[k]}
