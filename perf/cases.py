"""Work that users of this framework have it do, as measurable cases.

A case is a dict of plain values; ``kind`` says which public entry point it
goes through:

  count     ptw.pagerank: visit counts of geometric walks (PageRank, and
            personalised PageRank when the walkers start at given sources)
  rwr       ptw.rwr: (start, end) pairs of walks with restart
  deepwalk  ptw.deepwalk: fixed-length first-order paths
  node2vec  ptw.node2vec: fixed-length second-order paths
  batch     ptw.ppr_batch: many personalised queries in one call
  serve     ptw.Server: queries submitted, then stepped until all are done
  build     ptw.Graph.from_edges + export_csr: an edge list to a CSR and back
  train     ptw.learned.MLP: the walker-budget model trained and applied

``graph`` is "rmat" (R-MAT 0.57/0.19/0.19, symmetrised and cleaned), "raw"
(the R-MAT edge list as generated: directed, with duplicates, self-loops,
dead ends and gaps in the names) or "chung_lu" (power law, any number of
vertices).  ``tune`` is "" for a graph as it comes from its constructor, or
launch parameters as the command line's --tune takes them.  ``out`` is
"device" (a CUDA tensor that the caller keeps) or "host" (the call's own
numpy array).
"""
import math

import numpy as np
import torch

import ptwalker_gb300 as ptw
from ptwalker_gb300 import learned

# What the autotuner settles on for R-MAT scale 24 on a GB300.
TUNED = "block=768,ilp=2,chunk=64,hot_k=8192,cache_hints=1,paths_ilp=2,paths_named=0,ext_columns=3"


def listed():
    return [
        # The smallest call: a few thousand walkers on a toy graph or a unit
        # of an interactive session, where launches and latency are all.
        dict(name="count_small", kind="count", graph="rmat", scale=10, edge_factor=16, per_vertex=1.0,
             start="per_vertex", sp=0.15, tune="", out="device"),
        # An ordinary PageRank call as the README shows it: an untuned graph
        # of some hundred thousand vertices, counts in a new numpy array, the
        # reference application's uniform starts.
        dict(name="count_medium", kind="count", graph="rmat", scale=18, edge_factor=16, per_vertex=1.0,
             start="uniform", sp=0.15, tune="", out="host"),
        # A large untuned graph, one walker per vertex, counts kept on the GPU.
        dict(name="count_large", kind="count", graph="rmat", scale=22, edge_factor=16, per_vertex=1.0,
             start="per_vertex", sp=0.15, tune="", out="device"),
        # The benchmark workload: scale 24, the launch tuned beforehand.
        dict(name="count_largest", kind="count", graph="rmat", scale=24, edge_factor=16, per_vertex=1.0,
             start="per_vertex", sp=0.15, tune=TUNED, out="device"),
        # Personalised PageRank of one vertex (the ppr application): every
        # walker starts at the same place.
        dict(name="ppr_one_source", kind="count", graph="rmat", scale=20, edge_factor=16, walkers=100_000,
             start="sources", n_sources=1, sp=0.15, tune="", out="device"),
        # Random walk with restart, endpoints of every walker (the RWR
        # application): short walks, one output record each.
        dict(name="rwr_pairs", kind="rwr", graph="rmat", scale=22, edge_factor=16, per_vertex=1.0,
             start="uniform", sp=0.5, tune="", out="device"),
        # A training corpus for embeddings: 80-vertex paths from every vertex.
        dict(name="deepwalk_corpus", kind="deepwalk", graph="rmat", scale=22, edge_factor=16, per_vertex=1.0,
             start="per_vertex", walk_len=80, tune="", out="device"),
        # The same with second-order walks (in-out search, p = 2, q = 0.5).
        dict(name="node2vec_corpus", kind="node2vec", graph="rmat", scale=20, edge_factor=16, per_vertex=1.0,
             start="per_vertex", walk_len=80, p=2.0, q=0.5, tune="", out="device"),
        # Batched personalised PageRank for a GPU consumer: full vectors,
        # budgets from 10^3 to 10^6 walkers.
        dict(name="batch_queries", kind="batch", graph="rmat", scale=20, edge_factor=16, queries=512,
             budget_min=1000, budget_max=1_000_000, sp=0.2, app="visits", top_k=0, tune="", out="device"),
        # An online service under load on a power-law graph: the 1,000 most
        # visited vertices of every query.
        dict(name="serve_top1000", kind="serve", graph="chung_lu", vertices=1_000_003, mean_degree=32.0, queries=300,
             budget_min=1000, budget_max=1_000_000, sp=0.2, app="visits", top_k=1000, tune="", out="host"),
        # Ingest: an edge list in host memory, symmetrised, to a graph on the
        # GPU and its CSR back in host memory.
        dict(name="build_undirected", kind="build", edges=8_000_003, names=3_000_000, undirected=True),
        # The learned-budget model: trained on a few thousand labelled
        # sources, then applied to them.
        dict(name="train_budgets", kind="train", samples=2000, batch=256, epochs=30),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _some_graph(rng, scale_min, scale_max):
    """A graph between R-MAT scale_min and scale_max in size."""
    g = rng.choice(["rmat", "rmat", "raw", "chung_lu"])
    if g == "chung_lu":
        # as many edges as R-MAT of that scale at edge factor 16 has, at most
        n = int(_log(rng, 0.6 * 2 ** scale_min, 0.5 * 2 ** scale_max)) | 1
        return dict(graph=g, vertices=n, mean_degree=round(rng.uniform(8.0, 32.0), 2))
    return dict(graph=g, scale=rng.randint(scale_min, scale_max), edge_factor=rng.randint(5, 16))


def draw(rng):
    kind = rng.choice(["count", "count", "count", "rwr", "deepwalk", "node2vec", "batch", "serve", "build", "train"])
    c = dict(kind=kind)
    if kind in ("count", "rwr"):
        c.update(_some_graph(rng, 10, 22))
        c["start"] = rng.choice(["per_vertex", "uniform", "sources"])
        if c["start"] == "sources":
            c["n_sources"] = rng.choice([1, 1, rng.randint(2, 50)])
            c["walkers"] = int(_log(rng, 1000, 1_000_000))
        else:
            c["per_vertex"] = round(_log(rng, 0.25, 1.0), 4)
        c["sp"] = round(rng.uniform(0.15, 0.5), 3)
        c["tune"] = rng.choice(["", "", TUNED])
        c["out"] = rng.choice(["device", "device", "host"])
    elif kind in ("deepwalk", "node2vec"):
        c.update(_some_graph(rng, 10, 22 if kind == "deepwalk" else 20))
        c["start"] = rng.choice(["per_vertex", "uniform"])
        c["per_vertex"] = round(_log(rng, 0.1, 1.0), 4)
        c["walk_len"] = rng.randint(5, 80)
        if kind == "node2vec":
            c["p"], c["q"] = rng.choice([(2.0, 0.5), (0.5, 2.0), (1.0, 1.0), (4.0, 0.25), (0.25, 4.0)])
        c["tune"] = rng.choice(["", "", TUNED])
        c["out"] = "device"
    elif kind in ("batch", "serve"):
        c.update(_some_graph(rng, 14, 20))
        c["queries"] = int(_log(rng, 8, 300))
        c["budget_min"] = int(_log(rng, 100, 2000))
        c["budget_max"] = int(_log(rng, 5000, 1_000_000))
        c["sp"] = round(rng.uniform(0.2, 0.5), 3)
        c["app"] = rng.choice(["visits", "visits", "endpoint"])
        c["top_k"] = rng.choice([0, 100, 1000])
        c["tune"] = rng.choice(["", "", TUNED])
        c["out"] = "host" if kind == "serve" or c["top_k"] and rng.random() < 0.5 else "device"
        if kind == "serve" and not c["top_k"]:
            c["budget_max"] = min(c["budget_max"], 50_000)
    elif kind == "build":
        c["edges"] = int(_log(rng, 1000, 8_000_000)) | 1
        c["names"] = max(64, int(c["edges"] * rng.uniform(0.05, 0.4)))
        c["undirected"] = rng.random() < 0.5
    else:
        c["samples"] = rng.randint(300, 2000)
        c["batch"] = rng.choice([64, 100, 256, 512])
        most = max(1, 230 * c["batch"] // c["samples"])  # as many steps as the listed case has, at most
        c["epochs"] = rng.randint(min(5, most), min(30, most))
    return c


# ---- sizes (estimates, for work()) ---------------------------------------------

def _graph_size(case):
    """About how many vertices and CSR entries the case's graph has."""
    if case["graph"] == "chung_lu":
        n = 0.9 * case["vertices"]
        return n, 0.8 * case["vertices"] * case["mean_degree"]
    s, ef = case["scale"], case["edge_factor"]
    keep = min(1.0, 0.88 - 0.025 * (s - 10))  # share of the 2^s ids with an edge
    if case["graph"] == "raw":
        return keep * 2 ** s, ef * 2.0 ** s
    return keep * 2 ** s, 2.0 * ef * 2 ** s * (0.68 + 0.021 * (s - 10))


def _walkers(case, n):
    return int(case["walkers"]) if "walkers" in case else max(1, int(case["per_vertex"] * n))


def _mean_budget(case):
    a, b = float(case["budget_min"]), float(case["budget_max"])
    return (b - a) / math.log(b / a) if b > a else a


def work(case):
    """Bytes and operations that one pass cannot do without.  A move reads at
    least one 32-byte sector of the columns, unless the graph is smaller than
    that in all; every output is written once."""
    kind = case["kind"]
    if kind == "train":
        per_sample = 2.0 * (8 * 64 + 64 * 64 + 64)
        x = case["samples"] * case["epochs"]
        return dict(bytes=4.0 * 9 * case["samples"] + 4.0 * 4801, flops=3.0 * per_sample * x)
    if kind == "build":
        e, n = case["edges"], min(case["names"], 2.0 * case["edges"])
        entries = e * (2 if case["undirected"] else 1)
        return dict(bytes=8.0 * e + 4.0 * entries + 12.0 * n, flops=0.0)
    n, m = _graph_size(case)
    if kind in ("count", "rwr"):
        w = _walkers(case, n)
        moves = w / case["sp"]
        out = 4.0 * n if kind == "count" else 8.0 * w
    elif kind in ("deepwalk", "node2vec"):
        w = _walkers(case, n)
        moves = w * float(case["walk_len"] - 1)
        out = 4.0 * w * case["walk_len"]
    else:
        w = case["queries"] * _mean_budget(case)
        moves = w / case["sp"]
        visits = (w + moves if case["app"] == "visits" else w) / case["queries"]
        per_query = min(0.5 * n, 0.5 * visits)
        if case["top_k"]:
            per_query = min(per_query, case["top_k"])
        out = 8.0 * case["queries"] * per_query
    return dict(bytes=min(32.0 * moves, 4.0 * m + 8.0 * n) + out, flops=0.0)


# ---- inputs ---------------------------------------------------------------------

def _graph(case):
    """A program's graph is loaded once: the same for every seed (what is
    asked of it is not)."""
    if case["graph"] == "chung_lu":
        g = ptw.Graph.chung_lu(case["vertices"], 2.1, case["mean_degree"], seed=1)
    else:
        g = ptw.Graph.rmat(case["scale"], case["edge_factor"], seed=1, clean=case["graph"] == "rmat")
    if case["tune"]:
        g.tune = ptw.Tune(**{k: int(v) for k, v in (kv.split("=") for kv in case["tune"].split(","))})
    return g


def _names(g, case, rng, count):
    """Names of `count` vertices drawn uniformly (with repeats)."""
    if case["graph"] == "raw":
        return g.export_csr()[0][rng.integers(0, g.n, count)]
    return rng.integers(0, g.n, count).astype(np.uint32)  # names are 0 .. n - 1


def _edges(case, seed):
    """An edge list with power-law endpoints over scattered names, on the
    host; every name occurs."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    e, names = case["edges"], case["names"]
    table = torch.randperm(4 * names, generator=gen, device="cuda")[:names]
    ends = []
    for k in range(2):
        u = torch.rand(e, generator=gen, device="cuda", dtype=torch.float64)
        x = table[(u.pow(2.5) * names).long().clamp_(max=names - 1)]
        if k == 0:
            x[torch.randperm(e, generator=gen, device="cuda")[:names]] = table
        ends.append(x.to(torch.int32).cpu().numpy().view(np.uint32))
    return ends


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    st = dict(case=case, seed=int(seed) + 1)
    if kind == "build":
        st["src"], st["dst"] = _edges(case, seed)
        return st
    if kind == "train":
        x = rng.normal(0.0, 1.0, (case["samples"], 8)).astype(np.float32)
        t = (x[:, 0] + np.sin(x[:, 1]) + 0.1 * rng.normal(0.0, 1.0, case["samples"])).astype(np.float32)
        st.update(x=x, t=t)
        return st
    g = st["graph"] = _graph(case)
    if kind in ("batch", "serve"):
        q = case["queries"]
        st["sources"] = _names(g, case, rng, q)
        lo, hi = math.log(case["budget_min"]), math.log(case["budget_max"])
        st["budgets"] = np.exp(np.random.default_rng(q).uniform(lo, hi, q)).astype(np.int64)  # the case's own
        # room for every list: a query has at most this many entries
        length = 1.0 / case["sp"] + 1.0 if case["app"] == "visits" else 1.0
        room = np.minimum(case["top_k"] or g.n, np.minimum(g.n, st["budgets"] * length * 1.2 + 200)).astype(np.int64)
        if case["out"] == "device":
            st["keep"] = [torch.zeros(k, dtype=d, device="cuda") for k, d in
                          ((q + 1, torch.int64), (int(room.sum()), torch.int32), (int(room.sum()), torch.int32))]
        else:
            st["keep"] = [np.zeros(k, dtype=d) for k, d in
                          ((q + 1, np.int64), (int(room.sum()), np.int32), (int(room.sum()), np.int32))]
        if kind == "serve":
            st["server"] = ptw.Server(g, sp=case["sp"], seed=st["seed"], app=case["app"], table_bytes=4 << 30,
                                      top_k=case["top_k"])
        return st
    w = st["walkers"] = _walkers(case, g.n)
    st["sources"] = _names(g, case, rng, case["n_sources"]) if case["start"] == "sources" else None
    st["out"] = None
    if case["out"] == "device":
        shape = {"count": (g.id_bound,), "rwr": (w, 2)}.get(kind) or (w, case["walk_len"])
        st["out"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    return st


# ---- one pass ---------------------------------------------------------------------

def _whole(*arrays):
    """Unsigned arrays as the signed ones of their width (views)."""
    if isinstance(arrays[0], torch.Tensor):
        return tuple(a.view(torch.int64 if a.element_size() == 8 else torch.int32) for a in arrays)
    return tuple(a.view(np.int64 if a.itemsize == 8 else np.int32) for a in arrays)


def _keep(st, offsets, names, counts):
    """The lists, copied into the caller's own buffers."""
    off, nm, ct = st["keep"]
    e = len(names)
    if isinstance(off, torch.Tensor):
        off.copy_(offsets)
        nm[:e].copy_(names)
        ct[:e].copy_(counts)
    else:
        off[:], nm[:e], ct[:e] = offsets, names, counts
    return off, nm, ct


def _serve(st):
    srv = st["server"]
    for q, (s, b) in enumerate(zip(st["sources"], st["budgets"])):
        srv.submit(s, b, q)
    res = sorted(srv.drain(), key=lambda r: r["query_id"])
    off = np.cumsum([0] + [len(r["names"]) for r in res])
    return _keep(st, off, *_whole(np.concatenate([r["names"] for r in res]), np.concatenate([r["counts"] for r in res])))


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "build":
        with ptw.Graph.from_edges(st["src"], st["dst"], as_undirected=case["undirected"]) as g:
            return _whole(*g.export_csr())
    if kind == "train":
        m = learned.MLP(seed=st["seed"])
        curve = m.train(st["x"], st["t"], epochs=case["epochs"], batch=case["batch"], lr=3e-3, seed=st["seed"])
        y = m.forward(st["x"])
        params, norm = m.params()
        m.close()
        return curve, y, params, norm
    if kind == "serve":
        return _serve(st)
    g = st["graph"]
    if kind == "batch":
        dev = case["out"] == "device"
        r = ptw.ppr_batch(g, st["sources"], st["budgets"], sp=case["sp"], seed=st["seed"], app=case["app"],
                          top_k=case["top_k"], device_results=dev)
        kept = _keep(st, *_whole(*((r.d_offsets, r.d_names, r.d_counts) if dev else (r.offsets, r.names, r.counts))))
        r.close()
        return kept
    kw = dict(seed=st["seed"], start=case["start"], sources=st["sources"], out=st["out"])
    if kind == "count":
        return ptw.pagerank(g, st["walkers"], case["sp"], **kw)
    if kind == "rwr":
        return ptw.rwr(g, st["walkers"], case["sp"], **kw)
    if kind == "deepwalk":
        return ptw.deepwalk(g, st["walkers"], case["walk_len"], **kw)
    return ptw.node2vec(g, st["walkers"], case["walk_len"], case["p"], case["q"], **kw)


# ---- the same in 64 bits -----------------------------------------------------------

def _exact_train(case, st):
    """The budget model's training in numpy, 64 bits throughout, from the
    model's own initial weights and in its order of the samples."""
    m = learned.MLP(seed=st["seed"])
    p = m.params()[0].astype(np.float64)
    m.close()
    x, t = st["x"].astype(np.float64), st["t"].astype(np.float64)
    mu, sd, tmu, tsd = x.mean(0), x.std(0), t.mean(), t.std()
    xn, tn = (x - mu) / sd, (t - tmu) / tsd
    cut = np.cumsum([0, 8 * 64, 64, 64 * 64, 64, 64, 1])

    def parts(v):
        a = [v[cut[i]:cut[i + 1]] for i in range(6)]
        return a[0].reshape(8, 64), a[1], a[2].reshape(64, 64), a[3], a[4], a[5]

    def forward(z):
        w1, b1, w2, b2, w3, b3 = parts(p)
        z1 = z @ w1 + b1
        a1 = np.maximum(z1, 0.0)
        z2 = a1 @ w2 + b2
        a2 = np.maximum(z2, 0.0)
        return z1, a1, z2, a2, a2 @ w3 + b3[0]

    n, batch, mask = case["samples"], min(case["batch"], case["samples"]), (1 << 64) - 1
    perm, rs = list(range(n)), (st["seed"] * 0x9E3779B97F4A7C15 + 1) & mask
    b1, b2, lr = float(np.float32(0.9)), float(np.float32(0.999)), float(np.float32(3e-3))
    mom, var, step, curve = np.zeros_like(p), np.zeros_like(p), 0, []
    for _ in range(case["epochs"]):
        for i in range(n - 1, 0, -1):
            rs = (rs * 6364136223846793005 + 1442695040888963407) & mask
            j = (rs >> 33) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        losses = []
        for b0 in range(0, n, batch):
            idx = perm[b0:b0 + batch]
            z1, a1, z2, a2, y = forward(xn[idx])
            _, _, w2, _, w3, _ = parts(p)
            d = y - tn[idx]
            losses.append(float(np.mean(d * d)))
            e = 2.0 * d / len(idx)
            g2 = np.where(z2 > 0.0, e[:, None] * w3, 0.0)
            g1 = np.where(z1 > 0.0, g2 @ w2.T, 0.0)
            g = np.concatenate([(xn[idx].T @ g1).ravel(), g1.sum(0), (a1.T @ g2).ravel(), g2.sum(0), a2.T @ e,
                                [e.sum()]])
            step += 1
            mom = b1 * mom + (1.0 - b1) * g
            var = b2 * var + (1.0 - b2) * g * g
            p = p - lr * (mom / (1.0 - b1 ** step)) / (np.sqrt(var / (1.0 - b2 ** step)) + 1e-8)
        curve.append(float(np.mean(losses)))
    y = forward(xn)[4] * tsd + tmu
    return np.array(curve), y, p, np.concatenate([mu, sd, [tmu, tsd]])


def exact(case, seed):
    """Only the trained model's outputs are computed numbers: all others are
    counts, ids and edges, whole numbers that stay as they are."""
    if case["kind"] != "train":
        return None
    return _exact_train(case, prepare(case, seed))
