"""Which kernels a call takes must not show in its result: graphs at the
edges of the rules that choose between the integer and the FP64 sums and
between launch shapes, against the oracle (bit for bit: every sum here is
exact in any order)."""

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import oracle as O
import pcc_gb300 as P
import pcc_graphs as G

pytestmark = pytest.mark.gpu


def _weighted(g, w_of):
    """g with symmetric weights w_of(min id, max id)."""
    src = np.repeat(np.arange(g.n), np.diff(g.offsets).astype(np.int64))
    a, b = np.minimum(src, g.neighbors), np.maximum(src, g.neighbors)
    return P.CsrGraph(g.offsets, g.neighbors, w_of(a, b).astype(np.float32))


def _same(ctx, g, cfg, modularity=False):
    dg, og = ctx.upload(g), O.OracleGraph(g)
    run = (P.modularity_cluster, O.modularity_cluster) if modularity else (P.correlation_cluster, O.correlation_cluster)
    lab, st = run[0](dg, cfg)
    want, sto = run[1](og, cfg)
    np.testing.assert_array_equal(lab, want)
    for key in ("edge_visits", "rounds", "levels", "refine_passes"):
        assert st[key] == sto[key], key
    dg.free()
    return st


@pytest.mark.parametrize("scale,move,res", [
    (1, P.NBHR_CLUSTER_MOVE, 0.3), (1, P.NBHR_MOVE, 0.3),
    (30000, P.ALL_MOVE, 0.3), (4000000, P.ALL_MOVE, 0.3),                   # self-loops alone above 2^22
    (4000000, P.NBHR_CLUSTER_MOVE, 1.2e6), (4000000, P.NBHR_MOVE, 1.2e6)])  # other weights too
def test_heavy_self_loops(ctx, scale, move, res):
    """Contracted levels whose self-loops exceed 2^22 while the other weights
    may not: the self-loops must not decide the arithmetic, nor the result."""
    g, block = G.sbm(1500, 12, 0.2, 0.01, 5)
    gw = _weighted(g, lambda a, b: np.where(block[a] == block[b], scale, 1) + (a + b) % 3)
    st = _same(ctx, gw, P.make_config(resolution=res, refine=True, move_method=move))
    assert st["levels"] >= 2


def _hubby(n=6000, seed=3):
    """A block model with vertices of degree 700, 1500, 3000 and 5000, so that
    every kernel shape below the split rows takes part."""
    g, _ = G.sbm(n, 30, 0.05, 0.002, seed)
    src = np.repeat(np.arange(n), np.diff(g.offsets).astype(np.int64))
    keep = src < g.neighbors
    s, d = [src[keep]], [g.neighbors[keep].astype(np.int64)]
    for hub, deg in ((0, 700), (1, 1500), (2, 3000), (3, 5000)):
        s.append(np.full(deg, hub)), d.append(np.arange(10, 10 + deg))
    return P.CsrGraph.from_edges(n, np.concatenate(s), np.concatenate(d))


def _unit_hash(a, b):
    h = (a.astype(np.uint64) * np.uint64(0x9E3779B97F4A7C15) + b.astype(np.uint64) * np.uint64(0xD6E8FEB86659FD93))
    return ((h ^ (h >> np.uint64(29))) * np.uint64(0xBF58476D1CE4E5B9) >> np.uint64(40)).astype(np.float64) / 2.0 ** 24


# Weights by what the fixed-point rule has to say of them, and whether sums of
# any order are exact (then hubs equal the oracle's bits as well).
WEIGHTS = {
    "quarters": (lambda a, b: np.floor(_unit_hash(a, b) * 16) / 4, True),                  # 32-bit sums of 2^-2
    "negative": (lambda a, b: np.floor(_unit_hash(a, b) * 64) / 8 - 3, True),              # 32 bits, both signs, zeros
    "big_ints": (lambda a, b: np.floor(_unit_hash(a, b) * 9e4) + 4.3e6 * ((a + b) % 97 == 0), True),  # above 2^22
    "wide_ints": (lambda a, b: np.floor(_unit_hash(a, b) * 2 ** 20) * 2.0 ** 16, True),     # 64-bit sums
    "uniform": (lambda a, b: 0.5 + _unit_hash(a, b), True),                                # 64-bit sums of 2^-24
    "signed": (lambda a, b: _unit_hash(a, b) * 2 - 0.75, True),                            # 64 bits, both signs
    "spread": (lambda a, b: 10.0 ** (_unit_hash(a, b) * 12 - 9), False),                   # too wide: FP64
}


@pytest.mark.parametrize("kind", list(WEIGHTS))
def test_fixed_point_best_moves(ctx, kind):
    """One best-move pass per weight kind: targets, values and moves are the
    oracle's bits; certified and exact decisions are checked against each
    other on the device."""
    w_of, exact = WEIGHTS[kind]
    g = _weighted(_hubby(), w_of)
    dg, og = ctx.upload(g), O.OracleGraph(g)
    scale = max(float(np.abs(g.weights).mean()), 1e-6)
    low = np.diff(g.offsets) <= 1000
    for clusters, res, off in ((6000, 0.3, 0.0), (40, 0.002, 0.0), (40, 0.05, 0.0), (3, 0.001, 0.5)):
        rng = np.random.default_rng(clusters)
        C = rng.integers(0, clusters, g.n).astype(np.uint32)
        k = rng.integers(1, 5, g.n).astype(np.float64)
        s = np.bincount(C, minlength=g.n).astype(np.uint32)
        K = np.bincount(C, weights=k, minlength=g.n)
        cfg = P.make_config(resolution=res * scale, edge_weight_offset=off * scale)
        t, v, m = P.best_moves(dg, cfg, C, s, k, K)
        to, vo, mo = O.best_moves(og, cfg, C, s, k, K)
        part = slice(None) if exact and off == 0.0 else low
        np.testing.assert_array_equal(t[part], to[part])
        np.testing.assert_array_equal(v[part].view(np.uint64), vo[part].view(np.uint64))
        np.testing.assert_array_equal(m[part], mo[part])
    dg.free()


@pytest.mark.parametrize("kind", [k for k in WEIGHTS if WEIGHTS[k][1]])
@pytest.mark.parametrize("modularity", [False, True])
def test_fixed_point_clusterings(ctx, kind, modularity):
    """Whole clusterings on the weights whose sums are exact: every label."""
    g = _weighted(_hubby(seed=4), WEIGHTS[kind][0])
    scale = max(float(np.abs(g.weights).mean()), 1e-6)
    for move, res in ((P.NBHR_CLUSTER_MOVE, 0.02), (P.NBHR_MOVE, 0.2)):
        cfg = P.make_config(resolution=1.0 if modularity else res * scale, refine=True, move_method=move)
        _same(ctx, g, cfg, modularity)


def _ring_of_cliques(cliques, size, extra=0):
    """cliques complete graphs of `size` vertices joined in a ring, and
    `extra` isolated vertices at the end."""
    s, d = [], []
    for c in range(cliques):
        i, j = np.triu_indices(size, 1)
        s.append(c * size + i), d.append(c * size + j)
    if cliques > 1:
        s.append(np.arange(cliques) * size), d.append((np.arange(1, cliques + 1) % cliques) * size + 1)
    return P.CsrGraph.from_edges(cliques * size + extra, np.concatenate(s), np.concatenate(d))


# Sizes at the edges of the one-kernel round loop: one CTA and several, one
# vertex, a last slice of ids that is not full, rows at the limits of the
# lane groups, warps, teams and CTA tables, and rows above 4096.
LOOP_GRAPHS = {
    "two": lambda: P.CsrGraph.from_edges(2, [0], [1]),
    "edgeless": lambda: P.CsrGraph.from_edges(37, [], []),
    "cliques5": lambda: _ring_of_cliques(7, 5),
    "cliques33": lambda: _ring_of_cliques(40, 33, extra=5),
    "cliques130": lambda: _ring_of_cliques(9, 130, extra=70001),
    "cliques258": lambda: _ring_of_cliques(6, 258),
    "clique1002": lambda: _ring_of_cliques(3, 1002),
    "hubby": lambda: _hubby(7001, 9),
    "star9000": lambda: P.CsrGraph.from_edges(9001, np.zeros(9000, np.int64), np.arange(1, 9001)),
    "rmat15": lambda: G.rmat(15, 12, seed=8),
}


@pytest.mark.parametrize("name", list(LOOP_GRAPHS))
@pytest.mark.parametrize("move", [P.NBHR_CLUSTER_MOVE, P.NBHR_MOVE, P.ALL_MOVE])
def test_one_kernel_rounds(ctx, name, move):
    """A level's rounds in one kernel: labels and every counter equal the
    oracle's, and the host-driven rounds'."""
    g = LOOP_GRAPHS[name]()
    for res, inner, modularity in ((0.02, 0, False), (0.7, 1, False), (1.0, 3, True)):
        if modularity and g.m == 0:
            continue
        cfg = P.make_config(resolution=res, refine=True, move_method=move, louvain_num_inner_iterations=inner)
        st = _same(ctx, g, cfg, modularity)
        ctx.set_detailed_timing(True)
        try:
            host = _same(ctx, g, cfg, modularity)
        finally:
            ctx.set_detailed_timing(False)
        for key in ("vertex_visits", "moves", "family_entries", "family_vertices", "objective"):
            assert st[key] == host[key], key


def test_one_kernel_rounds_given_labels(ctx):
    """Rounds started from the caller's labels (isolated vertices included),
    with node weights and with 64-bit sums."""
    g, _ = G.sbm(3000, 20, 0.05, 0.002, 3)
    g = P.CsrGraph.from_edges(3100, np.repeat(np.arange(3000), np.diff(g.offsets).astype(np.int64)),
                              g.neighbors.astype(np.int64), symmetrize=False)
    rng = np.random.default_rng(2)
    init = rng.integers(0, 150, g.n).astype(np.uint32)
    for kind in (None, "uniform"):
        gw = g if kind is None else _weighted(g, WEIGHTS[kind][0])
        dg, og = ctx.upload(gw), O.OracleGraph(gw)
        for move in (P.NBHR_CLUSTER_MOVE, P.ALL_MOVE):
            cfg = P.make_config(resolution=0.05, refine=True, move_method=move)
            k = rng.integers(1, 4, g.n).astype(np.float64)
            lab, st = P.correlation_cluster(dg, cfg, k, init)
            want, so = O.correlation_cluster(og, cfg, k, init)
            np.testing.assert_array_equal(lab, want)
            assert (st["rounds"], st["edge_visits"]) == (so["rounds"], so["edge_visits"])
        dg.free()


@pytest.mark.parametrize("name", ["two", "cliques33", "clique1002", "hubby", "star9000", "rmat15"])
@pytest.mark.parametrize("weights", ["unit", "integer"])
def test_whole_cluster_moves_table(ctx, name, weights):
    """Whole-cluster moves summed in the (cluster, cluster) table, rounds on
    the device and driven by the host: singletons (every sum one entry), given
    labels of few clusters (few sums, many entries), negative values."""
    g = LOOP_GRAPHS[name]()
    if weights == "integer":
        g = _weighted(g, lambda a, b: (a * 7 + b * 13) % 5 + 1)
    dg, og = ctx.upload(g), O.OracleGraph(g)
    rng = np.random.default_rng(4)
    for res, offset, move, groups in ((0.02, 0.0, P.NBHR_CLUSTER_MOVE, 0), (0.5, 2.0, P.NBHR_MOVE, 3),
                                      (0.1, 0.0, P.ALL_MOVE, 40)):
        init = rng.integers(0, min(groups, g.n), g.n).astype(np.uint32) if groups else None
        cfg = P.make_config(resolution=res, edge_weight_offset=offset, move_method=move, num_iterations=6,
                            clustering_moves_method=P.DEFAULT_CLUSTER_MOVES)
        want, so = O.correlation_cluster(og, cfg, None, init)
        for detailed in (False, True):
            ctx.set_detailed_timing(detailed)
            try:
                lab, st = P.correlation_cluster(dg, cfg, None, init)
            finally:
                ctx.set_detailed_timing(False)
            np.testing.assert_array_equal(lab, want)
            for key in ("edge_visits", "rounds", "levels", "moves"):
                assert st[key] == so[key], key
    dg.free()


def _hub_degrees(degs, n=9000, seed=6):
    """A block model with one hub of each given degree (its ids first)."""
    g, _ = G.sbm(n, 30, 0.03, 0.001, seed)
    src = np.repeat(np.arange(n), np.diff(g.offsets).astype(np.int64))
    far = (src >= len(degs)) & (g.neighbors >= len(degs)) & (src < g.neighbors)
    s, d = [src[far]], [g.neighbors[far].astype(np.int64)]
    rng = np.random.default_rng(seed)
    for hub, deg in enumerate(degs):
        s.append(np.full(deg, hub)), d.append(len(degs) + rng.permutation(n - len(degs))[:deg])
    return P.CsrGraph.from_edges(n, np.concatenate(s), np.concatenate(d))


@pytest.mark.parametrize("kind", ["unit", "integer", "uniform", "wide"])
@pytest.mark.parametrize("move", [P.NBHR_CLUSTER_MOVE, P.ALL_MOVE])
def test_hubs_at_table_edges(ctx, kind, move):
    """Hubs at the limits of the table sizes, the degree-binned kernels driven
    by the host; their rows are pushed whole and in pieces."""
    g = _hub_degrees((1000, 1001, 2047, 2048, 3071, 4096, 4097, 6144, 6145, 8500))
    if kind == "integer":
        g = _weighted(g, lambda a, b: (a * 7 + b * 13) % 5 + 1)
    elif kind == "uniform":
        g = _weighted(g, WEIGHTS["uniform"][0])
    elif kind == "wide":
        g = _weighted(g, lambda a, b: ((a * 7 + b * 13) % 5 + 1) * 1000003)
    scale = float(np.abs(g.weights).mean()) if g.weights is not None else 1.0
    ctx.set_detailed_timing(True)
    try:
        for res, modularity in ((0.02 * scale, False), (1.0, True)):
            _same(ctx, g, P.make_config(resolution=res, refine=True, move_method=move), modularity)
    finally:
        ctx.set_detailed_timing(False)


@pytest.mark.parametrize("kind", ["unit", "uniform"])
def test_one_partition_hubs(ctx, kind):
    """Hubs of one table of 16,384 slots, up to its last degree and beyond."""
    g = _hub_degrees((4097, 8191, 8192, 12287, 12288, 12289, 24576, 24577), n=26000)
    if kind == "uniform":
        g = _weighted(g, WEIGHTS["uniform"][0])
    ctx.set_detailed_timing(True)
    try:
        for res, modularity in ((0.005, False), (1.0, True)):
            _same(ctx, g, P.make_config(resolution=res, refine=True, move_method=P.NBHR_CLUSTER_MOVE), modularity)
    finally:
        ctx.set_detailed_timing(False)


@pytest.mark.parametrize("labels", ["one", "own", "sparse"])
def test_modularity_of_given_labels(ctx, labels):
    """Labels of any spacing: one cluster, singletons, ids far apart."""
    g = _hub_degrees((1001, 4097, 8500))
    dg, og = ctx.upload(g), O.OracleGraph(g)
    rng = np.random.default_rng(1)
    lab = {"one": np.full(g.n, g.n - 1), "own": np.arange(g.n)[::-1].copy(),
           "sparse": rng.permutation(g.n)[:37][rng.integers(0, 37, g.n)]}[labels].astype(np.uint32)
    dense = np.unique(lab, return_inverse=True)[1].astype(np.uint32)
    assert P.modularity(dg, 0.7, lab) == pytest.approx(O.modularity(og, 0.7, dense), rel=1e-12, abs=1e-12)
    dg.free()


def test_graph_shared_by_contexts(ctx):
    """One resident graph clustered by two contexts at once, from two threads:
    whichever call builds the graph's hub plan and the bins of its isolated
    vertices, the other finds them complete."""
    degs = (1500, 4097, 9000, 13000, 40000)
    g = _hub_degrees(degs, n=45000)
    g = P.CsrGraph(np.concatenate([g.offsets, np.full(70, g.offsets[-1])]), g.neighbors)  # isolated vertices
    init = np.random.default_rng(5).integers(0, 300, g.n).astype(np.uint32)
    cfg = P.make_config(resolution=0.01, refine=True)
    want = O.correlation_cluster(O.OracleGraph(g), cfg, None, init)[0]
    other = P.Context(0)
    try:
        for _ in range(6):
            dg = ctx.upload(g)
            view = P.DeviceGraph(other, dg.handle)
            try:
                with ThreadPoolExecutor(2) as pool:
                    got = list(pool.map(lambda v: P.correlation_cluster(v, cfg, None, init)[0], (dg, view)))
            finally:
                view._h = None  # the graph is dg's to free
            dg.free()
            for lab in got:
                np.testing.assert_array_equal(lab, want)
    finally:
        other.close()


@pytest.mark.parametrize("name", ["hubby", "rmat15", "cliques130"])
def test_round_kernel_gives_up(ctx, monkeypatch, name):
    """A grid barrier whose bounded wait runs out (a limit of no polls: every
    CTA leaves at its first barrier): the call answers INTERNAL, calls that
    need no barrier go on working on that context, and other contexts give
    the oracle's labels afterwards."""
    monkeypatch.setenv("PCC_BARRIER_POLLS", "0")
    short = P.Context(0)
    monkeypatch.delenv("PCC_BARRIER_POLLS")
    g = LOOP_GRAPHS[name]()
    cfg = P.make_config(resolution=0.05, refine=True)
    try:
        dg = short.upload(g)
        for _ in range(2):
            with pytest.raises(P.PccError) as e:
                P.correlation_cluster(dg, cfg)
            assert e.value.code == 13 and "error flag 5" in str(e.value)
        short.set_detailed_timing(True)  # rounds without the round kernel
        np.testing.assert_array_equal(P.correlation_cluster(dg, cfg)[0], O.correlation_cluster(O.OracleGraph(g), cfg)[0])
        short.set_detailed_timing(False)
        _same(short, P.CsrGraph.from_edges(2, [0], [1]), cfg)  # one CTA: no barrier to wait at
        dg.free()
    finally:
        short.close()
    _same(ctx, g, cfg)


def test_tuned_context_keeps_round_kernel(ctx):
    """A launch shape set on the context is for the degree-binned kernels: a
    level that fits the round kernel takes it all the same (with the same few
    launches), and switching it off takes none of the results."""
    g, _ = G.sbm(3000, 30, 0.04, 0.001, 42)
    dg = ctx.upload(g)
    cfg = P.make_config(resolution=0.05, refine=True)
    lab, st = P.correlation_cluster(dg, cfg)
    try:
        ctx.set_launch_tuning(16, 256, 0.5)
        tuned, tuned_st = P.correlation_cluster(dg, cfg)
        ctx.set_round_kernel(False)
        binned, binned_st = P.correlation_cluster(dg, cfg)
    finally:
        ctx.set_round_kernel(True)
        ctx.set_launch_tuning(0, 0, 0.0)
    for other in (tuned, binned):
        np.testing.assert_array_equal(lab, other)
    assert tuned_st["kernel_launches"] == st["kernel_launches"]
    assert binned_st["kernel_launches"] > 2 * st["kernel_launches"]
    for key in ("rounds", "edge_visits", "vertex_visits", "moves", "objective"):
        assert st[key] == tuned_st[key] == binned_st[key], key
    # (The shape moves degrees 17-32 to the warp family of the binned kernels.)
    assert st["family_entries"] == tuned_st["family_entries"]
    assert sum(st["family_entries"]) == sum(binned_st["family_entries"])
    dg.free()


@pytest.mark.parametrize("name", ["hubby", "rmat15"])
@pytest.mark.parametrize("shape", [(4, 1000, 1.0), (8, 512, 0.5), (16, 256, 2.0), (32, 128, 0.125), (32, 64, 4.0)])
def test_launch_shapes_without_round_kernel(ctx, name, shape):
    """The accepted launch shapes on the degree-binned kernels in the graph
    loop, 32-bit and 64-bit sums."""
    g = LOOP_GRAPHS[name]()
    try:
        ctx.set_round_kernel(False)
        ctx.set_launch_tuning(*shape)
        for gw, res in ((g, 0.02), (_weighted(g, WEIGHTS["uniform"][0]), 0.02)):
            _same(ctx, gw, P.make_config(resolution=res, refine=True, move_method=P.NBHR_MOVE))
    finally:
        ctx.set_round_kernel(True)
        ctx.set_launch_tuning(0, 0, 0.0)


def _peak(c, run):
    """Device bytes that run() took beyond what the context held."""
    held = c.bytes_in_use()
    c.lib.pcc_device_peak_bytes(c.handle, 1)
    out = run()
    return c.lib.pcc_device_peak_bytes(c.handle, 0) - held, out


def test_no_round_kernel_tables_elsewhere(ctx):
    """A call that cannot enter the round kernel takes none of its hub tables
    (24 bytes an entry of every row above 4096 entries): a best-move pass holds
    some arrays of up to 8 bytes a vertex, 128 bytes in all, and small lists."""
    g = _hub_degrees((8000,) * 60)
    dg = ctx.upload(g)
    C = np.arange(g.n, dtype=np.uint32)
    one = np.ones(g.n)
    cfg = P.make_config(resolution=0.1)
    peak, _ = _peak(ctx, lambda: P.best_moves(dg, cfg, C, C * 0 + 1, one, one))
    assert peak <= 128 * g.n + (2 << 20) < 24 * 60 * 8000
    dg.free()


BUDGET_GRAPHS = {
    "hubs": lambda: _hub_degrees((8000,) * 60),
    "rmat15": LOOP_GRAPHS["rmat15"],
    "real": lambda: _weighted(_hubby(seed=4), WEIGHTS["uniform"][0]),
}


@pytest.mark.parametrize("name", list(BUDGET_GRAPHS))
@pytest.mark.parametrize("modularity", [False, True])
def test_round_kernel_within_a_budget(ctx, name, modularity):
    """A budget that the degree-binned kernels just fit is enough with the round
    kernel on: levels that it has no memory for run without it."""
    g = BUDGET_GRAPHS[name]()
    cfg = P.make_config(resolution=1.0 if modularity else 0.02, refine=True)

    def call(budget, kernel=True):
        c = P.Context(0, budget)
        try:
            c.set_round_kernel(kernel)
            return _peak(c, lambda: P.cluster_host_csr(c, g, cfg, objective=int(modularity)))
        finally:
            c.close()

    binned, (want, _) = call(1 << 38, False)
    free, (lab, _) = call(1 << 38)
    np.testing.assert_array_equal(lab, want)
    for budget in np.linspace(binned, max(free, binned), 5).astype(int).tolist():
        _, (lab, _) = call(budget)
        np.testing.assert_array_equal(lab, want)
    with pytest.raises(P.PccError) as e:
        call(binned // 2)
    assert e.value.code == 8


@pytest.mark.parametrize("clusters", [200, 60000, 300000])  # 1, 2 and 3 passes of the vertex sort
def test_contraction_frees_what_is_spent(built, clusters):
    """Peak of a contraction under a budget, where arrays are freed as they are
    spent: the vertex sort's spare buffers (12 bytes a vertex) are not held
    beyond the sort, whichever of the two the result lies in."""
    n = 300000
    ring = np.arange(n)
    g = P.CsrGraph.from_edges(n, ring, (ring + 1) % n)
    C = (ring % clusters).astype(np.uint32)
    c = P.Context(0, 1 << 38)
    try:
        dg = c.upload(g)
        peak, out = _peak(c, lambda: P.compress(dg, C, np.ones(n)))
        m2 = out.info()[1]
        # Per vertex: 12 labels and node weights, 4 ids of the clusters, then
        # 4 ranks, 12 sorted vertices, 12 spare, 8 row starts; per new vertex 12
        # offset and count; per cluster 8 segment start, 20 class lists and count;
        # per entry 8 moved; per new entry 8.
        rows, r = (12 + 4) * n + 12 * clusters, clusters
        held = max(rows + (4 + 12 + 12) * n, rows + (4 + 12 + 8) * n + 8 * r, rows + (4 + 8) * n + 8 * r + 8 * g.m,
                   rows + 28 * r + 8 * g.m + 8 * m2)
        assert peak <= held + (1 << 20)
        out.free()
        dg.free()
    finally:
        c.close()


@pytest.mark.parametrize("name", ["sbm", "hubby"])
def test_cluster_move_table_within_a_budget(built, name):
    """Whole-cluster moves take their table when all of it fits, and give it
    back before the scores are computed: a budget that the sorted path needs
    (the same graph with weights that are no integers) is enough,
    and a call that succeeds under a budget does under every larger one."""
    g = G.sbm(20000, 40, 0.02, 0.0004, 4)[0] if name == "sbm" else _hubby()
    gw = _weighted(g, lambda a, b: 1.5 + 0 * a)
    cfg = P.make_config(resolution=0.1, clustering_moves_method=P.DEFAULT_CLUSTER_MOVES)
    want = O.correlation_cluster(O.OracleGraph(g), cfg)[0]

    def call(budget, graph=g):
        c = P.Context(0, budget)
        try:
            peak, (lab, _) = _peak(c, lambda: P.cluster_host_csr(c, graph, cfg))
        except P.PccError as e:
            assert e.code == 8
            return None
        finally:
            c.close()
        if graph is g:
            np.testing.assert_array_equal(lab, want)
        return peak

    sorted_path = call(1 << 38, gw) - 4 * g.m  # (weights are 4 bytes an entry)
    assert call(sorted_path) is not None
    full = call(1 << 38)
    fits = [call(b) is not None for b in np.linspace(full - 24 * g.m - 32 * g.n, full, 60).astype(int).tolist()]
    assert fits[-1] and fits == sorted(fits)


def _split_hubs():
    """Hubs of every kind: one CTA, one, two and four partitions."""
    return _hub_degrees((1500, 4097, 9000, 13000, 40000), n=45000)


FP64_CALLS = {  # graph, weights, resolution, offset: no fixed point holds these sums
    "spread_sbm": (lambda: G.sbm(3000, 20, 0.05, 0.002, 3)[0], "spread", 0.1, 0.0),
    "spread_lfr": (lambda: G.lfr(20000, mean_degree=20, dmax=900, seed=9)[0], "spread", 0.1, 0.0),
    "offset_lfr": (lambda: G.lfr(20000, mean_degree=20, dmax=900, seed=9)[0], "uniform", 0.1, 0.3),
    "offset_unit": (lambda: G.sbm(3000, 20, 0.05, 0.002, 3)[0], None, 0.02, 0.25),
    "spread_hubs": (_split_hubs, "spread", 0.01, 0.0),
    "offset_hubs": (_split_hubs, "uniform", 0.01, 0.3),
}


@pytest.mark.parametrize("name", list(FP64_CALLS))
@pytest.mark.parametrize("move", [P.NBHR_CLUSTER_MOVE, P.NBHR_MOVE])
def test_fp64_clusterings(ctx, name, move):
    """Whole synchronous clusterings on the FP64 kernels, in the graph loop and
    driven by the host.  On the block models every row of every level is short,
    its sums have the reference's order and every label is the oracle's; rows
    above 1000 entries add in any order, as the reference's do, so there the
    labels agree to 99.9% and the objective to 1e-9."""
    make, kind, res, off = FP64_CALLS[name]
    g = make()
    if kind:
        g = _weighted(g, WEIGHTS[kind][0])
    scale = float(np.abs(g.weights).mean()) if kind else 1.0
    cfg = P.make_config(resolution=res * scale, edge_weight_offset=off, refine=True, move_method=move)
    dg, og = ctx.upload(g), O.OracleGraph(g)
    want, so = O.correlation_cluster(og, cfg)
    for detailed in (False, True):
        ctx.set_detailed_timing(detailed)
        try:
            lab, st = P.correlation_cluster(dg, cfg)
        finally:
            ctx.set_detailed_timing(False)
        assert st["objective"] == pytest.approx(so["objective"], rel=1e-9)
        if not name.endswith(("sbm", "unit")):
            assert np.mean(lab == want) >= 0.999
        else:
            np.testing.assert_array_equal(lab, want)
            assert (st["rounds"], st["edge_visits"], st["levels"]) == (so["rounds"], so["edge_visits"], so["levels"])
    dg.free()


@pytest.mark.parametrize("name", ["hubby", "rmat15", "split_hubs", "clique1002"])
@pytest.mark.parametrize("kind", ["unit", "uniform"])
@pytest.mark.parametrize("move", [P.NBHR_CLUSTER_MOVE, P.NBHR_MOVE, P.ALL_MOVE])
def test_graph_loop_without_round_kernel(ctx, name, kind, move):
    """The degree-binned kernels in the graph loop, families on branches and one
    after another, on levels that the round kernel takes by default: labels
    and counters equal the round kernel's."""
    g = _split_hubs() if name == "split_hubs" else LOOP_GRAPHS[name]()
    if kind != "unit":
        g = _weighted(g, WEIGHTS[kind][0])
    cfg = P.make_config(resolution=0.02, refine=True, move_method=move, louvain_num_iterations=6,
                        louvain_num_inner_iterations=5)
    with pytest.MonkeyPatch.context() as mp:
        mp.setenv("PCC_SERIAL_FAMILIES", "1")
        serial = P.Context(0)
    out = []
    try:
        for c, kernel in ((ctx, True), (ctx, False), (serial, True)):
            c.set_round_kernel(kernel)
            dg = c.upload(g)
            out.append(P.correlation_cluster(dg, cfg))
            dg.free()
    finally:
        ctx.set_round_kernel(True)
        serial.close()
    for lab, st in out[1:]:
        np.testing.assert_array_equal(lab, out[0][0])
        assert st["kernel_launches"] > out[0][1]["kernel_launches"]
        for key in ("objective", "num_clusters", "levels", "rounds", "refine_passes", "edge_visits", "vertex_visits",
                    "moves", "family_entries", "family_vertices"):
            assert st[key] == out[0][1][key], key


def _clique_moves(ctx, size, w_of, res):
    """A best-move pass and a clustering of one clique with the given weights
    (and a few isolated vertices), against the oracle's bits."""
    g = _weighted(_ring_of_cliques(1, size, extra=9), w_of)
    dg, og = ctx.upload(g), O.OracleGraph(g)
    rng = np.random.default_rng(size)
    one = np.ones(g.n)
    for clusters in (1, 2, 7, g.n):
        C = rng.integers(0, clusters, g.n).astype(np.uint32)
        s, K = np.bincount(C, minlength=g.n).astype(np.uint32), np.bincount(C, minlength=g.n).astype(np.float64)
        cfg = P.make_config(resolution=res)
        for got, exp in zip(P.best_moves(dg, cfg, C, s, one, K), O.best_moves(og, cfg, C, s, one, K)):
            np.testing.assert_array_equal(got.view(np.uint64 if got.dtype == np.float64 else got.dtype),
                                          exp.view(np.uint64 if exp.dtype == np.float64 else exp.dtype))
    dg.free()
    _same(ctx, g, P.make_config(resolution=res, refine=True))


@pytest.mark.parametrize("size,weight", [
    (256, 2.0 ** 22), (257, 2.0 ** 22),                          # integers: rows of 2^30 - 2^22 and 2^30
    (128, 2.0 ** 22 + 0.5), (129, 2.0 ** 22 + 0.5),              # halves: just below and above 2^30 units
    (256, 2.0 ** 44), (257, 2.0 ** 44),                          # beside weights of 1: below and at 2^52
    (256, 2.0 ** 14), (257, 2.0 ** 14)])                         # beside weights of 2^-30: below and at 2^52 units
@pytest.mark.parametrize("sign", [1, -1, 0])
def test_sums_at_the_limits(ctx, size, weight, sign):
    """Rows whose sums lie right below and above the lines between 32-bit and
    64-bit sums and between those and FP64; both signs, and mixed ones."""
    small = {2.0 ** 44: 1.0, 2.0 ** 14: 2.0 ** -30}.get(weight)

    def w_of(a, b):
        w = np.full(a.shape, weight)
        if small:
            w[(a * 31 + b * 17) % 11 == 0] = small
        return w * (sign if sign else np.where((a + b) % 2, 1.0, -1.0))

    _clique_moves(ctx, size, w_of, 0.3 * weight)


@pytest.mark.parametrize("kind", ["subnormal", "zero", "least", "negative_zero"])
def test_tiny_weights(ctx, kind):
    """Subnormal weights, the smallest one among ones, and zeros of both signs."""
    w_of = {"subnormal": lambda a, b: np.ldexp(1.0 + (a * 7 + b * 13) % 5, -149),
            "least": lambda a, b: np.where((a + b) % 9 == 0, np.ldexp(1.0, -149), 1.0),
            "zero": lambda a, b: 0.0 * a,
            "negative_zero": lambda a, b: np.where((a + b) % 3 == 0, -0.0, 2.0)}[kind]
    _clique_moves(ctx, 70, w_of, {"subnormal": 1e-45, "least": 0.4, "zero": 0.4, "negative_zero": 0.4}[kind])


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_rows_beside_infinite_and_nan_weights(ctx, value):
    """One edge of infinite or undefined weight decides nothing for the rows that
    do not hold it."""
    g = _hubby()
    far = g.neighbors[g.offsets[20]]
    g = _weighted(g, lambda a, b: np.where((np.minimum(20, far) == a) & (np.maximum(20, far) == b), value,
                                           1.0 + (a + b) % 4))
    rows = np.repeat(np.arange(g.n), np.diff(g.offsets).astype(np.int64))
    odd = np.unique(rows[~np.isfinite(g.weights)])
    assert odd.size == 2
    low = (np.diff(g.offsets) <= 1000) & ~np.isin(np.arange(g.n), odd)
    dg, og = ctx.upload(g), O.OracleGraph(g)
    C = np.random.default_rng(1).integers(0, 40, g.n).astype(np.uint32)
    one = np.ones(g.n)
    s, K = np.bincount(C, minlength=g.n).astype(np.uint32), np.bincount(C, minlength=g.n).astype(np.float64)
    cfg = P.make_config(resolution=0.02)
    for got, exp in zip(P.best_moves(dg, cfg, C, s, one, K), O.best_moves(og, cfg, C, s, one, K)):
        np.testing.assert_array_equal(got[low], exp[low])
    dg.free()
