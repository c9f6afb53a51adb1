"""What a user of the engine has it do, as cases to time: one-at-a-time and
batched matching on the benchmark's resident graphs, unlabeled pattern
counting, loading a graph and answering the first query, the reference-layout
transforms, and a training step of the order network.

Graphs and queries are the repository's own workloads
(fsig_gb300/workloads.py): the data graph of a matching case is the resident
handle that a serving program keeps, so it is built and loaded once per
process; the queries come from the seed.  ``listed``, ``draw``, ``prepare``,
``run``, ``work`` and ``exact`` are the whole interface.
"""
from __future__ import annotations

import json
import math

import numpy as np

import fsig_gb300 as F
from fsig_gb300 import learn
from fsig_gb300 import workloads as W

ALGOS = {"fsig": F.ALGO_FSIG, "gsi": F.ALGO_GSI, "fused": F.ALGO_FUSED}

# (vertices, adjacency entries, labels) of the resident graphs
SHAPES = {"c1": (10_000, 100_000, 8), "c2": (320_000, 2_100_000, 16), "c4": (320_000, 2_100_000, 16),
          "c5": (1 << 22, 1 << 27, 32)}


def listed():
    return [
        # One small query on a small graph, one call: a user at the command
        # line or a service with single requests.  Latency and launches count.
        {"name": "match_c1", "kind": "match", "graph": "c1", "queries": 1, "algo": "gsi"},
        # Mid-scale graph, one eight-vertex query per call (the plain serving
        # path), with the neighbour-support refinement of algorithm 1.
        {"name": "match_c2", "kind": "match", "graph": "c2", "queries": 8, "algo": "fsig"},
        # The largest graph, one 12-32-vertex query per call.
        {"name": "match_c5", "kind": "match", "graph": "c5", "queries": 4, "algo": "fused"},
        # A batch of small queries on a small graph.
        {"name": "batch_c1", "kind": "batch", "graph": "c1", "queries": 100, "algo": "fused", "learned": False,
         "use_graph": False, "refine": -1},
        # A batch of eight-vertex queries, dense and sparse, signature filter only.
        {"name": "batch_c2", "kind": "batch", "graph": "c2", "queries": 200, "algo": "gsi", "learned": False,
         "use_graph": False, "refine": -1},
        # Serving: uneven queries of 4-32 vertices, 512 per CUDA graph, learned order.
        {"name": "batch_c4", "kind": "batch", "graph": "c4", "queries": 512, "algo": "fused", "learned": True,
         "use_graph": True, "refine": -1},
        # The benchmark's headline: 512 queries of 12-32 vertices on 2^26 edges.
        {"name": "batch_c5", "kind": "batch", "graph": "c5", "queries": 512, "algo": "fused", "learned": True,
         "use_graph": True, "refine": -1},
        # An odd, small batch on the largest graph with all filters and refinement.
        {"name": "batch_c5_refined", "kind": "batch", "graph": "c5", "queries": 37, "algo": "fused",
         "learned": False, "use_graph": False, "refine": 2},
        # Unlabeled counting of a five-vertex pattern on a skewed graph.
        {"name": "pattern_house", "kind": "pattern", "vertices": 700, "pattern": "house"},
        # Cold start: load a large labelled graph and answer a first query.
        {"name": "load_large", "kind": "load", "vertices": 1 << 20, "edges": 1 << 24, "labels": 16},
        # The reference's transformers in a row: CSR, signatures, PCSR.
        {"name": "transforms", "kind": "transforms", "vertices": 320_000, "edges": 1_050_000, "labels": 4},
        # One minibatch of the order network's training (learn.train's size).
        {"name": "train_step", "kind": "train", "graphs": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["match", "match", "batch", "batch", "batch", "pattern", "load", "transforms", "train"])
    if kind == "match":
        graph = rng.choice(["c1", "c2", "c5"])
        algo = rng.choice(["fsig", "gsi", "fused"]) if graph != "c5" else "fused"
        return {"kind": kind, "graph": graph, "queries": _log_int(rng, 1, 12), "algo": algo}
    if kind == "batch":
        graph = rng.choice(["c1", "c2", "c4", "c5"])
        learned = rng.random() < 0.5
        return {"kind": kind, "graph": graph, "queries": _log_int(rng, 2, {"c1": 100, "c2": 200}.get(graph, 500)),
                "algo": "fused", "learned": learned, "use_graph": rng.random() < 0.5,
                "refine": rng.choice([-1, -1, 1, 2])}
    if kind == "pattern":
        return {"kind": kind, "vertices": _log_int(rng, 100, 800), "pattern": rng.choice(sorted(W.PATTERNS))}
    if kind == "load":
        v = _log_int(rng, 10_000, 1 << 20)
        return {"kind": kind, "vertices": v, "edges": int(v * rng.uniform(3.0, 16.0)), "labels": rng.randint(8, 32)}
    if kind == "transforms":
        v = _log_int(rng, 10_000, 400_000)
        return {"kind": kind, "vertices": v, "edges": int(v * rng.uniform(2.0, 5.0)), "labels": rng.randint(2, 4)}
    return {"kind": kind, "graphs": _log_int(rng, 16, 2048)}


# ---------------------------------------------------------------------------
# resident graphs and their queries
# ---------------------------------------------------------------------------
_RESIDENT = {}
_SPECS = {}


def _resident(name):
    """(engine with the graph loaded and the packaged network, graph, csr)."""
    key = "c2" if name == "c4" else name
    if key not in _RESIDENT:
        g = W.build_graph(key)
        e = F.Engine(0, arena_bytes=(24 if key == "c5" else 8) << 30)
        e.load_graph(g)
        e.mpnn_set_params(learn.load_params())
        _RESIDENT[key] = (e, g, g.csr())
    return _RESIDENT[key]


def _manifest(name):
    """Generator specs of the workload's queries in ascending order of their
    recorded work, those of its tuning batch, and the mean embedding count."""
    if name not in _SPECS:
        m = json.loads(W.manifest_path(name).read_text())
        specs = [tuple(s) for b in m["batches"] for s in b["specs"]]
        work = [x for b in m["batches"] for x in b["work"]]
        counts = [x for b in m["batches"] for x in b["counts"]]
        order = sorted(range(len(specs)), key=lambda i: (work[i], i))
        _SPECS[name] = ([specs[i] for i in order], [tuple(s) for s in m["tune_specs"]],
                        float(np.mean(np.asarray(counts, np.float64))))
    return _SPECS[name]


def _queries(name, count, rng):
    """`count` of the workload's queries.  A small sample takes one from the
    middle of each of `count` classes of recorded work, so that two samples
    cost about the same; a large one is drawn from all queries."""
    ranked, tune, _ = _manifest(name)
    n = len(ranked)
    if 2 * count <= n:
        edges = np.linspace(0, n, count + 1)
        picked = [ranked[min(n - 1, int(a + (b - a) * (0.25 + 0.5 * rng.random())))]
                  for a, b in zip(edges[:-1], edges[1:])]
    else:
        pool = ranked + tune
        picked = [pool[i] for i in rng.choice(len(pool), count, replace=False)]
    picked = [picked[i] for i in rng.permutation(len(picked))]
    _, g, csr = _resident(name)
    return F.gen_queries(g, picked, csr=csr)


def _labelled_rmat(v, e, labels, seed):
    return F.gen_rmat(v, e, 0.57, 0.19, 0.19, seed=seed, labels=F.gen_labels(v, labels, "zipf", seed=seed))


def _renumbered_chung_lu(v, e, labels, seed):
    """One power-law graph under vertex numbers and an edge order of the
    seed's choice (so the sizes of its PCSR units do not depend on the seed)."""
    g = F.gen_chung_lu(v, e, 2.1, seed=2, labels=F.gen_labels(v, labels, "zipf", seed=2))
    rng = np.random.default_rng(seed)
    number = rng.permutation(v).astype(np.uint32)
    lab = np.empty_like(g.labels)
    lab[number] = g.labels
    return F.Graph(lab, number[g.edges[rng.permutation(e)]])


def _train_inputs(graphs, seed):
    """Random connected query graphs of 4-32 vertices with their features,
    neighbour masks and targets (a vertex's position in an order)."""
    rng = np.random.default_rng(seed)
    sizes = rng.integers(4, 33, graphs)
    goff = np.zeros(graphs + 1, np.uint32)
    goff[1:] = np.cumsum(sizes)
    total = int(goff[-1])
    nbr = np.zeros(total, np.uint32)
    tgt = np.zeros(total, np.float32)
    for g, n in enumerate(sizes.tolist()):
        o = int(goff[g])
        pairs = [(i, int(rng.integers(0, i))) for i in range(1, n)]
        pairs += [tuple(int(x) for x in p) for p in rng.integers(0, n, (n, 2))]
        for a, b in pairs:
            if a != b:
                nbr[o + a] |= np.uint32(1 << b)
                nbr[o + b] |= np.uint32(1 << a)
        tgt[o:o + n] = rng.permutation(n) / max(n - 1, 1)
    feat = rng.random((total, F.MPNN_FEATURES)).astype(np.float32)
    params = learn.init_params(seed % (1 << 31))
    params[learn.P_BIN:learn.P_WS] = rng.normal(0, 0.1, learn.H)
    params[learn.P_B:learn.P_WOUT] = rng.normal(0, 0.1, learn.LAYERS * learn.H)
    return goff, feat, nbr, tgt, params


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("match", "batch"):
        e, _, _ = _resident(case["graph"])
        return {"case": case, "engine": e, "queries": _queries(case["graph"], case["queries"], rng)}
    if kind == "pattern":
        v = case["vertices"]
        e = F.Engine(0, arena_bytes=2 << 30)
        e.load_graph(F.gen_rmat(v, 16 * v, 0.57, 0.19, 0.19, seed=int(seed)))
        return {"case": case, "engine": e, "query": W.pattern(case["pattern"])}
    if kind == "load":
        g = _labelled_rmat(case["vertices"], case["edges"], case["labels"], int(seed))
        n = case["labels"]
        # a path through three rare labels
        q = F.Query(np.array([n - 1, n - 2, n - 3], np.int32), np.array([[0, 1], [1, 2]], np.uint32))
        return {"case": case, "engine": F.Engine(0, arena_bytes=4 << 30), "graph": g, "query": q}
    if kind == "transforms":
        g = _renumbered_chung_lu(case["vertices"], case["edges"], case["labels"], int(seed))
        return {"case": case, "engine": F.Engine(0, arena_bytes=4 << 30), "graph": g}
    goff, feat, nbr, tgt, params = _train_inputs(case["graphs"], int(seed))
    e = F.Engine(0, arena_bytes=1 << 30)
    e.mpnn_set_params(params)
    return {"case": case, "engine": e, "data": (goff, feat, nbr, tgt)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _rows(lists):
    out = np.zeros((len(lists), F.MAX_QUERY), np.int64)
    for row, x in zip(out, lists):
        row[:len(x)] = x
    return out


def _outputs(rs):
    """Every result whole, one row per query."""
    return {"count": np.array([r.count for r in rs], np.int64),
            "hash": np.array([r.hash for r in rs], np.uint64).view(np.int64),
            "status": np.array([r.status for r in rs], np.int32),
            "order": _rows([r.order for r in rs]),
            "candidates": _rows([r.candidates for r in rs]),
            "levels": _rows([r.level_counts for r in rs])}


def run(state):
    case, e = state["case"], state["engine"]
    kind = case["kind"]
    if kind == "match":
        algo = ALGOS[case["algo"]]
        return _outputs([e.match(q, algo) for q in state["queries"]])
    if kind == "batch":
        kw = dict(algo=ALGOS[case["algo"]], refine_iters=case["refine"], use_graph=case["use_graph"])
        if case["learned"]:
            # serving in learned order: a query over the work limit runs again in heuristic order
            rs, _ = learn.match_learned(e, state["queries"], work_limit=W.WORK_BUDGET, **kw)
        else:
            rs = e.match_batch(state["queries"], **kw)
        return _outputs(rs)
    if kind == "pattern":
        return _outputs([e.match(state["query"], F.ALGO_GSI)])
    if kind == "load":
        e.load_graph(state["graph"])
        out = _outputs([e.match(state["query"], F.ALGO_GSI)])
        out.update(e.graph_info())
        return out
    if kind == "transforms":
        g = state["graph"]
        off, adj = e.build_csr(g.num_vertices, g.edges)
        sig = e.build_signature(g.labels, off, adj, column_oriented=True)
        units = e.build_pcsr(g.labels, off, adj, case["labels"])
        return {"offsets": off.view(np.int32), "adjacency": adj.view(np.int32), "signature": sig.view(np.int32),
                "units": [(k, m, table.view(np.int32), lists.view(np.int32)) for k, m, table, lists in units]}
    loss, grads = e.mpnn_train_step(*state["data"], lr=2e-3)
    return {"loss": loss, "grads": grads}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
HASH_OPS = 30  # integer operations of the two 64-bit mixes every embedding's hash takes


def work(case):
    """Bytes: the graph (labels, offsets, adjacency) read once and the results
    written once; operations: the hash of every embedding, or the network's
    products."""
    kind = case["kind"]
    if kind in ("match", "batch"):
        v, a, _ = SHAPES[case["graph"]]
        n = case["queries"]
        return {"bytes": 8 * v + 4 * a + 700 * n, "flops": HASH_OPS * _manifest(case["graph"])[2] * n}
    if kind == "pattern":
        return {"bytes": 8 * case["vertices"] + 8 * 16 * case["vertices"], "flops": 0}
    if kind == "load":
        # edges and labels in; offsets, adjacency and 64-byte signatures out
        return {"bytes": 16 * case["edges"] + 72 * case["vertices"], "flops": 0}
    if kind == "transforms":
        # edges and labels in; CSR, signatures and PCSR lists out (the slot tables depend on the graph)
        return {"bytes": 24 * case["edges"] + 72 * case["vertices"], "flops": 0}
    nodes = 18 * case["graphs"]
    products = 16 * 64 + 6 * 64 * 64
    return {"bytes": nodes * 44 + 8 * learn.N_PARAMS, "flops": 6 * nodes * products}


def exact(case, seed):
    """The training step's loss and gradients in 64 bits; matching, loading
    and the transforms return whole numbers, which have no nearer value."""
    if case["kind"] != "train":
        return None
    import torch
    goff, feat, nbr, tgt, params = _train_inputs(case["graphs"], int(seed))
    total = int(goff[-1])
    rows, cols = [], []
    owner = np.repeat(goff[:-1].astype(np.int64), np.diff(goff.astype(np.int64)))
    for w in range(32):
        hit = np.nonzero((nbr >> np.uint32(w)) & np.uint32(1))[0]
        rows.append(hit)
        cols.append(owner[hit] + w)
    rows, cols = torch.from_numpy(np.concatenate(rows)), torch.from_numpy(np.concatenate(cols))
    deg = torch.zeros(total, dtype=torch.float64).index_add_(0, rows, torch.ones(len(rows), dtype=torch.float64))
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1.0), torch.zeros_like(deg))[:, None]
    p = torch.tensor(params, dtype=torch.float64, requires_grad=True)
    h, layers = learn.H, learn.LAYERS
    w_in = p[learn.P_WIN:learn.P_BIN].reshape(learn.F_PAD, h)
    w_s = p[learn.P_WS:learn.P_WN].reshape(layers, h, h)
    w_n = p[learn.P_WN:learn.P_B].reshape(layers, h, h)
    b = p[learn.P_B:learn.P_WOUT].reshape(layers, h)
    x = torch.zeros(total, learn.F_PAD, dtype=torch.float64)
    x[:, :learn.F_IN] = torch.from_numpy(feat.astype(np.float64))
    a = torch.relu(x @ w_in + p[learn.P_BIN:learn.P_WS])
    for i in range(layers):
        mean = torch.zeros_like(a).index_add(0, rows, a[cols]) * inv
        a = torch.relu(a @ w_s[i] + mean @ w_n[i] + b[i])
    score = a @ p[learn.P_WOUT:learn.P_BOUT] + p[learn.P_BOUT]
    loss = ((score - torch.from_numpy(tgt.astype(np.float64))) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad.numpy()}
