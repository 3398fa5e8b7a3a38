"""The clustering calls whose time is watched: small, ordinary and large graphs
through the package's public entry points, with the objectives, move methods,
weights and ways in (resident graph, host buffers, batch, server, text) that
users call them with.

Asynchronous moves are not among them: their results differ from run to run by
design, so two versions cannot be held against each other.
"""

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "parallel-correlation-clustering_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import pcc_gb300 as P  # noqa: E402
import pcc_graphs as G  # noqa: E402

MOVES = {"nbhr_cluster": P.NBHR_CLUSTER_MOVE, "all": P.ALL_MOVE, "nbhr": P.NBHR_MOVE}


def listed():
    return [
        # The low end of the batched workload's sizes, called one graph at a
        # time: launches and host work are everything.
        {"name": "sbm_300_correlation", "way": "resident", "graph": "sbm", "n": 300, "blocks": 6, "degree": 12.0,
         "objective": "correlation", "resolution": 0.05, "move": "nbhr_cluster"},
        # The seeded stochastic block model that the CPU clusterer is run on:
        # every vertex in every round.
        {"name": "sbm_10k_all_moves", "way": "resident", "graph": "sbm", "n": 10000, "blocks": 50, "degree": 15.0,
         "objective": "correlation", "resolution": 0.01, "move": "all"},
        # The high end of the batched workload's sizes, modularity with the
        # default move method: an ordinary community graph.
        {"name": "sbm_50k_modularity", "way": "resident", "graph": "sbm", "n": 49999, "blocks": 100, "degree": 20.0,
         "objective": "modularity", "resolution": 1.0, "move": "nbhr_cluster"},
        # A power-law graph that a program has in host memory: upload,
        # clustering and labels back in one call.
        {"name": "rmat_18_host_buffers", "way": "host", "graph": "rmat", "n": 262144, "factor": 16,
         "objective": "modularity", "resolution": 1.0, "move": "nbhr"},
        # The benchmark's workload: RMAT scale 22, synchronous modularity.
        {"name": "rmat_22_modularity", "way": "resident", "graph": "rmat", "n": 4194304, "factor": 16,
         "objective": "modularity", "resolution": 1.0, "move": "nbhr"},
        # The serving mix's heavy request: correlation barely contracts it, so
        # every level is about as large as the first.
        {"name": "rmat_20_correlation", "way": "resident", "graph": "rmat", "n": 1048576, "factor": 16,
         "objective": "correlation", "resolution": 0.1, "move": "nbhr_cluster"},
        # LFR-like graph with real edge weights: sums in 64-bit floats.
        {"name": "lfr_1m_real_weights", "way": "resident", "graph": "lfr", "n": 1000003, "degree": 20.0, "weights": "real",
         "objective": "correlation", "resolution": 0.1, "move": "nbhr_cluster"},
        # Integer weights and whole-cluster moves after each round.
        {"name": "sbm_120k_cluster_moves", "way": "resident", "graph": "sbm", "n": 120001, "blocks": 100, "degree": 16.0,
         "weights": "integer", "method": "cluster_moves", "refine": False,
         "objective": "correlation", "resolution": 0.05, "move": "nbhr_cluster"},
        # Many independent graphs of uneven size in one call.
        {"name": "batch_128", "way": "batch", "count": 128, "resolution": 0.05},
        # A burst of requests on the server: mostly small block models, one in
        # twenty an RMAT graph of scale 20, mixed resolutions and objectives.
        {"name": "serve_40", "way": "serve", "count": 40, "rmat_n": 1048576, "rmats": 2},
        # Scoring of a clustering that the caller has: objective, modularity
        # and the comparison with known communities.
        {"name": "score_lfr_500k", "way": "score", "graph": "lfr", "n": 500009, "degree": 20.0, "weights": "real",
         "resolution": 0.1},
        # What the command line does: adjacency text in, clustering text out.
        {"name": "text_sbm_100k", "way": "text", "graph": "sbm", "n": 100003, "blocks": 120, "degree": 16.0,
         "objective": "correlation", "resolution": 0.05, "move": "nbhr_cluster"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    way = rng.choice(["resident", "resident", "resident", "resident", "resident", "resident", "host", "batch", "serve",
                      "score", "text"])
    if way == "batch":
        return {"way": way, "count": _log(rng, 4, 128), "resolution": rng.choice([0.01, 0.05, 0.2])}
    if way == "serve":
        return {"way": way, "count": _log(rng, 4, 40), "rmat_n": _log(rng, 1 << 15, 1 << 20), "rmats": rng.randint(0, 2)}
    c = {"way": way, "graph": rng.choice(["sbm", "rmat", "lfr"])}
    if way == "text":
        c["graph"] = "sbm"
    if way == "score":
        c["graph"] = "lfr"
    if c["graph"] == "sbm":
        c["n"] = _log(rng, 200, 100000 if way == "text" else 150000)
        c["blocks"] = rng.randint(2, max(2, min(200, c["n"] // 8)))
        c["degree"] = rng.uniform(8.0, 32.0)
        if way == "resident":
            c["weights"] = rng.choice(["unit", "unit", "integer", "real"])
            c["given_labels"] = rng.random() < 0.15  # RefineClusters from the caller's labels
    elif c["graph"] == "rmat":
        c["n"] = _log(rng, 1 << 12, 3 << 20 if way == "resident" else 1 << 19)
        c["factor"] = rng.randint(6, 16)
    else:
        c["n"] = _log(rng, 5000, 600000 if way == "resident" else 500000)
        c["degree"] = rng.uniform(12.0, 24.0)
        c["weights"] = rng.choice(["real", "real", "unit"])
    if way == "score":
        c["resolution"] = rng.choice([0.01, 0.1, 0.5])
        return c
    c["objective"] = rng.choice(["correlation", "modularity"])
    # Correlation work on a hub-heavy graph grows with its size much faster
    # than modularity work, which contracts it.
    if c["graph"] == "rmat" and c["objective"] == "correlation":
        c["n"] = min(c["n"], 1 << 19)
    c["resolution"] = 1.0 if c["objective"] == "modularity" else rng.choice([0.01, 0.05, 0.1, 0.5])
    c["move"] = rng.choice(["nbhr_cluster", "nbhr", "nbhr", "all"])
    if way == "resident":
        c["refine"] = rng.random() < 0.8
        if c["graph"] == "sbm" and rng.random() < 0.15:
            c["method"] = "cluster_moves"
            c["refine"] = False
    return c


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _rmat(n, factor, seed):
    """RMAT (0.57 / 0.19 / 0.19 / 0.05) on n vertices: ids of the next power of
    two, those of n and above dropped; symmetric, no repeats or self-loops."""
    scale = max(1, (n - 1).bit_length())
    count = factor * n
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.zeros(count, dtype=torch.int64, device="cuda")
    v = torch.zeros(count, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        x = torch.rand(count, generator=gen, device="cuda")
        u.mul_(2).add_(x >= 0.76)
        v.mul_(2).add_(((x >= 0.57) & (x < 0.76)) | (x >= 0.95))
    keep = (u != v) & (u < n) & (v < n)
    u, v = u[keep], v[keep]
    key = torch.unique(torch.cat([u * n + v, v * n + u]))
    del u, v, keep
    src = key // n
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    nbr = (key - src * n).to(torch.int32).cpu().numpy().view(np.uint32)
    return P.CsrGraph(off.cpu().numpy().astype(np.uint64), nbr)


def _graph(case, seed):
    """(CsrGraph, planted community of each vertex or None)."""
    n, kind, weights = case["n"], case["graph"], case.get("weights", "unit")
    if kind == "rmat":
        return _rmat(n, case["factor"], seed), None
    if kind == "sbm":
        # As the batched workload: p_out / p_in = 0.02 at the given mean degree.
        size = n / case["blocks"]
        p_in = min(1.0, case["degree"] / max((size - 1.0) + 0.02 * (n - size), 1e-9))
        g, truth = G.sbm(n, case["blocks"], p_in, 0.02 * p_in, seed)
    else:
        lo, hi = (0.5, 1.5) if weights == "real" else (0.0, 0.0)
        g, truth = G.lfr(n, case["degree"], min(2000, n // 4), cmax=min(5000, n // 4), w_lo=lo, w_hi=hi, seed=seed)
        return (g if weights == "real" else P.CsrGraph(g.offsets, g.neighbors)), truth
    if weights != "unit":
        src = np.repeat(np.arange(n, dtype=np.uint64), np.diff(g.offsets).astype(np.int64))
        dst = g.neighbors.astype(np.uint64)
        h = (np.minimum(src, dst) * np.uint64(0x9E3779B97F4A7C15) + np.maximum(src, dst) * np.uint64(0xD6E8FEB86659FD93)
             + np.uint64(seed)) >> np.uint64(40)
        w = 1 + h % np.uint64(5) if weights == "integer" else 0.5 + h.astype(np.float64) / 2.0 ** 24
        g = P.CsrGraph(g.offsets, g.neighbors, w.astype(np.float32))
    return g, truth


def _config(case):
    moves = P.DEFAULT_CLUSTER_MOVES if case.get("method") == "cluster_moves" else P.LOUVAIN
    # permute orders the asynchronous rounds only; the LFR workload sets it.
    return P.make_config(resolution=case["resolution"], refine=case.get("refine", True),
                         move_method=MOVES[case.get("move", "nbhr_cluster")], clustering_moves_method=moves,
                         permute=case.get("graph") == "lfr")


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    count, rmats = case["count"], min(case["rmats"], case["count"])
    at = set(np.random.default_rng(count).choice(count, rmats, replace=False).tolist())
    out = []
    for i, (n, b, pi, po, _) in enumerate(G.batch_sbm_spec(count, 12)):
        heavy = i in at
        g = _rmat(case["rmat_n"], 16, seed * 1000 + i) if heavy else G.sbm(n, b, pi, po, seed * 1000 + i)[0]
        # One heavy request of each objective; the small ones at random.
        objective = len([j for j in at if j < i]) % 2 if heavy else int(rng.integers(0, 2))
        cfg = P.make_config(resolution=0.1 if heavy else float(rng.choice([0.01, 0.1, 0.5])), refine=True)
        out.append((g, cfg, objective))
    return out


_shared = {}


def _context():
    """The one context that a program keeps."""
    if "ctx" not in _shared:
        _shared["ctx"] = P.Context(0)
    return _shared["ctx"]


def _server():
    """The one server that a serving program keeps: 8 slots, 120 GB."""
    if "server" not in _shared:
        _shared["server"] = P.Server(8, 120 << 30)
    return _shared["server"]


def _labels_near(truth, n, seed):
    """The planted communities with one vertex in ten moved: what a caller
    has from an earlier run."""
    rng = np.random.default_rng(seed)
    lab = truth.astype(np.uint32).copy()
    wrong = rng.random(n) < 0.1
    lab[wrong] = rng.integers(0, int(lab.max()) + 1, int(wrong.sum()), dtype=np.uint32)
    return lab


def _communities(truth, n):
    """The largest planted communities, as ground-truth files list them (a
    top-5000 file): offsets and members."""
    sizes = np.bincount(truth)
    top = np.argsort(-sizes, kind="stable")[:min(5000, n // 100)]
    order = np.argsort(truth, kind="stable")
    start = np.concatenate([[0], np.cumsum(sizes)])
    members = np.concatenate([order[start[c]:start[c + 1]] for c in top]).astype(np.uint32)
    off = np.zeros(top.size + 1, np.uint64)
    off[1:] = np.cumsum(sizes[top])
    return off, members


def prepare(case, seed):
    way = case["way"]
    if way == "batch":
        # The workload's sizes, with edges from the seed.
        spec = G.batch_sbm_spec(case["count"], 7)
        return {"way": way, "graphs": [G.sbm(n, b, pi, po, seed * 1000 + i)[0] for i, (n, b, pi, po, _) in enumerate(spec)],
                "cfg": P.make_config(resolution=case["resolution"], refine=True)}
    if way == "serve":
        return {"way": way, "server": _server(), "requests": _requests(case, seed)}
    ctx = _context()
    g, truth = _graph(case, seed)
    s = {"way": way, "ctx": ctx, "cfg": _config(case), "modularity": case.get("objective") == "modularity"}
    if way == "host":
        s["host"] = g
    elif way == "text":
        s["text"] = ("AdjacencyGraph\n%d\n%d\n" % (g.n, g.m) + "\n".join(map(str, g.offsets[:-1].tolist())) + "\n"
                     + "\n".join(map(str, g.neighbors.tolist())) + "\n").encode()
    else:
        s["graph"] = ctx.upload(g)
        if case.get("given_labels") or way == "score":
            s["labels"] = _labels_near(truth, g.n, seed)
    if way == "score":
        s["offsets"], s["members"] = _communities(truth, g.n)
        s["resolution"] = case["resolution"]
    return s


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------
def _result(labels, stats, modularity):
    return {"labels": labels.view(np.int32), "clusters": stats["num_clusters"], "rounds": stats["rounds"],
            "objective": stats["modularity"] if modularity else stats["objective"]}


def run(state):
    way = state["way"]
    if way == "batch":
        labels, stats, _ = P.cluster_batch(state["graphs"], state["cfg"])
        return {"labels": np.concatenate(labels).view(np.int32), "clusters": np.array([s["num_clusters"] for s in stats]),
                "objectives": np.array([s["objective"] for s in stats])}
    if way == "serve":
        srv = state["server"]
        tickets = [srv.submit(g, cfg, obj) for g, cfg, obj in state["requests"]]
        got = [srv.wait(t) for t in tickets]
        return {"labels": np.concatenate([x[0] for x in got]).view(np.int32), "clusters": np.array([x[1]["num_clusters"] for x in got]),
                "objectives": np.array([x[1]["objective"] for x in got]),
                "modularities": np.array([x[1]["modularity"] for x in got])}
    ctx, cfg = state["ctx"], state["cfg"]
    if way == "score":
        g, lab = state["graph"], state["labels"]
        scores, prec, rec = P.compare_communities(ctx, lab, offsets=state["offsets"], members=state["members"])
        return {"objective": P.objective(g, cfg, lab), "modularity": P.modularity(g, state["resolution"], lab),
                "precision": prec, "recall": rec, "average": np.array([scores["avg_precision"], scores["avg_recall"]])}
    if way == "host":
        labels, stats = P.cluster_host_csr(ctx, state["host"], cfg, 1 if state["modularity"] else 0)
        return _result(labels, stats, state["modularity"])
    if way == "text":
        g = ctx.parse_gbbs(state["text"], False)
        labels, stats = P.modularity_cluster(g, cfg) if state["modularity"] else P.correlation_cluster(g, cfg)
        g.free()
        text = ctx.format_clustering(labels)
        # In a buffer of the longest text that n ids can give.
        out = np.zeros(labels.size * (len(str(labels.size)) + 2), np.uint8)
        out[:len(text)] = np.frombuffer(text, np.uint8)
        return {"text": out, **_result(labels, stats, state["modularity"])}
    if state["modularity"]:
        labels, stats = P.modularity_cluster(state["graph"], cfg, state.get("labels"))
    else:
        labels, stats = P.correlation_cluster(state["graph"], cfg, None, state.get("labels"))
    return _result(labels, stats, state["modularity"])


def work(case):
    """The graph read once and the labels written once (text: its bytes once
    each way); the number of rounds is the data's own."""
    way = case["way"]
    small = 9000 * 4 + 9000 * 20 * 4 + 9000 * 8  # a batched block model: 9,000 vertices of degree 20 in the mean
    if way == "batch":
        return {"bytes": case["count"] * small, "flops": 0}
    if way == "serve":
        return {"bytes": (case["count"] - case["rmats"]) * small + case["rmats"] * case["rmat_n"] * (12 + 4 * 30),
                "flops": 0}
    n = case["n"]
    m = n * (2 * case["factor"] * 0.94 if case["graph"] == "rmat" else case["degree"])
    weighted = case.get("weights", "unit") != "unit"
    graph = 8 * (n + 1) + m * (8 if weighted else 4)
    if way == "text":
        digits = len(str(n)) + 0.5
        return {"bytes": n * (digits + 1) + m * digits + n * digits, "flops": 0}
    if way == "score":
        return {"bytes": 2 * graph + 3 * 4 * n, "flops": 2 * m}
    return {"bytes": graph + 4 * n, "flops": 0}


def exact(case, seed):
    """Scores in 64 bits.  The clusterings have no such value: their objective
    is that of the labels that the call itself finds."""
    if case["way"] != "score":
        return None
    g, truth = _graph(case, seed)
    lab = _labels_near(truth, g.n, seed)
    src = np.repeat(np.arange(g.n), np.diff(g.offsets).astype(np.int64))
    same = lab[src] == lab[g.neighbors]
    w = np.ones(g.m) if g.weights is None else g.weights.astype(np.float64)
    sizes = np.bincount(lab).astype(np.float64)
    res = case["resolution"]
    objective = math.fsum(w[same]) / 2 - res / 2 * float((sizes * (sizes - 1)).sum())
    deg = np.bincount(lab, weights=np.diff(g.offsets).astype(np.float64))
    modularity = (float(same.sum()) - res * float((deg * deg).sum()) / g.m) / g.m
    # Communities against clusters: the largest intersection, the lowest
    # cluster among equals.
    off, members = _communities(truth, g.n)
    count = off.size - 1
    com = np.repeat(np.arange(count), np.diff(off).astype(np.int64))
    k = int(lab.max()) + 1
    pair, hits = np.unique(com * k + lab[members], return_counts=True)
    com, clu = pair // k, pair % k
    order = np.lexsort((clu, -hits, com))
    com, clu, hits = com[order], clu[order], hits[order].astype(np.float64)
    first = np.ones(com.size, bool)
    first[1:] = com[1:] != com[:-1]
    precision = hits[first] / sizes[clu[first]]
    recall = hits[first] / np.diff(off).astype(np.float64)
    return {"objective": objective, "modularity": modularity, "precision": precision, "recall": recall,
            "average": np.array([precision.mean(), recall.mean()])}
