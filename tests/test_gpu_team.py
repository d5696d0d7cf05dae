"""Phases that a team of thread blocks runs in one kernel, against the CPU
oracle, at the sizes where the team changes form (one block, a cluster, a
cooperative grid; 256 vertices per block), at the row lengths where a lane, a
warp or a block takes over (32, 256, 1024) and at the limits of its rule (1024
blocks for the dense counters; 8192 blocks and rows of 2048 entries for the
hash tables), just past which the per-step launches take over.  Integer
outputs: equality.
"""
import numpy as np
import pytest

from conftest import csr_from_edges

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def N():
    from kahip_b200 import native
    assert native.device_count() > 0, "no CUDA device"
    return native


@pytest.fixture(scope="module")
def O():
    from oracle import oracle
    return oracle


def weighted(g, seed):
    rng = np.random.default_rng(seed)
    g["vwgt"] = rng.integers(0, 6, g["n"]).astype(np.int32)
    src = np.repeat(np.arange(g["n"]), np.diff(g["xadj"]))
    lo, hi = np.minimum(src, g["adjncy"]).astype(np.int64), np.maximum(src, g["adjncy"]).astype(np.int64)
    g["adjwgt"] = ((lo * 31 + hi * 17 + seed) % 7).astype(np.int32)  # zero weights among them
    return g


def hub_graph(n, hub, seed):
    """A ring, one vertex of `hub` neighbours and some of 100-400."""
    rng = np.random.default_rng(seed)
    edges = {(v, v + 1) for v in range(1, n - 1)}
    edges |= {(0, v) for v in range(1, hub + 1)}
    for c in (5, 900):
        edges |= {(min(c, int(u)), max(c, int(u))) for u in rng.choice(np.arange(1000, n), 100 + 300 * (c > 5), False)}
    return csr_from_edges(n, sorted(edges))


def skewed(n, k, seed):
    """Most vertices in the first blocks: the balance repair has work."""
    rng = np.random.default_rng(seed)
    p = np.minimum(rng.integers(0, k, n), rng.integers(0, k, n)).astype(np.int32)
    return p


SIZES = [1, 31, 255, 256, 257, 511, 513, 1024, 2047, 2048, 2049, 4096, 4097, 8192, 40001, 160000]
HUBS = [32, 33, 128, 129, 256, 257, 1024, 1025, 2048, 2049]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("k", [2, 13])
def test_jet_sizes(N, O, graphs, n, k):
    g = graphs.rgg2d(n, seed=n) if n > 31 else csr_from_edges(n, [(i, i + 1) for i in range(n - 1)])
    for unit in (True, False):
        if not unit:
            weighted(g, n)
        kn_o, kn_p = O.knobs(g, k, 0.03, 5, 1), N.derive_knobs(n, g["vwgt"], k, 0.03, 5, 1)
        part = skewed(n, k, n)
        for level in (0, 1):
            assert np.array_equal(O.jet_refine(g, kn_o, part, kn_o.upper_bound, level),
                                  N.jet_refine(g, kn_p, part, kn_p.upper_bound, level))


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("k", [9, 64])
def test_refine_sizes(N, O, graphs, n, k):
    g = graphs.rgg3d(n, seed=n) if n > 31 else csr_from_edges(n, [(i, i + 1) for i in range(n - 1)])
    for unit in (True, False):
        if not unit:
            weighted(g, n)
        kn_o, kn_p = O.knobs(g, k, 0.03, 5, 0), N.derive_knobs(n, g["vwgt"], k, 0.03, 5, 0)
        part = skewed(n, k, n)
        bal_o, ok_o = O.balance(g, kn_o, part, kn_o.upper_bound, 1)
        bal_p, ok_p = N.balance(g, kn_p, part, kn_p.upper_bound, 1)
        assert ok_o == ok_p and np.array_equal(bal_o, bal_p)
        assert np.array_equal(O.lp_refine(g, kn_o, bal_o, kn_o.upper_bound, 1),
                              N.lp_refine(g, kn_p, bal_o, kn_p.upper_bound, 1))


@pytest.mark.parametrize("hub", HUBS)
@pytest.mark.parametrize("k", [40, 1025])
def test_refine_hubs(N, O, hub, k):
    g = hub_graph(5000, hub, hub)
    for unit in (True, False):
        if not unit:
            weighted(g, hub)
        kn_o, kn_p = O.knobs(g, k, 0.10, 1, 0), N.derive_knobs(g["n"], g["vwgt"], k, 0.10, 1, 0)
        part = skewed(g["n"], k, hub)
        bal_o, ok_o = O.balance(g, kn_o, part, kn_o.upper_bound, 1)
        bal_p, ok_p = N.balance(g, kn_p, part, kn_p.upper_bound, 1)
        assert ok_o == ok_p and np.array_equal(bal_o, bal_p)
        assert np.array_equal(O.lp_refine(g, kn_o, bal_o, kn_o.upper_bound, 1),
                              N.lp_refine(g, kn_p, bal_o, kn_p.upper_bound, 1))


@pytest.mark.parametrize("hub", HUBS)
def test_jet_hubs(N, O, hub):
    g = hub_graph(5000, hub, hub)
    for k in (2, 40, 1025):
        kn_o, kn_p = O.knobs(g, k, 0.03, 1, 1), N.derive_knobs(g["n"], g["vwgt"], k, 0.03, 1, 1)
        part = skewed(g["n"], k, hub)
        assert np.array_equal(O.jet_refine(g, kn_o, part, kn_o.upper_bound, 1),
                              N.jet_refine(g, kn_p, part, kn_p.upper_bound, 1))


@pytest.mark.parametrize("k", [1024, 1025, 8192, 8193])
def test_jet_many_blocks(N, O, graphs, k):
    g = graphs.rgg2d(20000, seed=2)
    kn_o, kn_p = O.knobs(g, k, 0.10, 1, 1), N.derive_knobs(g["n"], g["vwgt"], k, 0.10, 1, 1)
    part = skewed(g["n"], k, 3)
    assert np.array_equal(O.jet_refine(g, kn_o, part, kn_o.upper_bound, 0),
                          N.jet_refine(g, kn_p, part, kn_p.upper_bound, 0))


@pytest.mark.parametrize("n", SIZES)
def test_cluster_sizes(N, O, graphs, n):
    g = graphs.rgg2d(n, seed=n) if n > 31 else csr_from_edges(n, [(i, i + 1) for i in range(n - 1)])
    for unit in (True, False):
        if not unit:
            weighted(g, n)
        for k in (2, 64):
            kn_o, kn_p = O.knobs(g, k, 0.03, 5, 0), N.derive_knobs(n, g["vwgt"], k, 0.03, 5, 0)
            for level in (0, 1):
                assert np.array_equal(O.lp_cluster(g, kn_o, level), N.lp_cluster(g, kn_p, level))


@pytest.mark.parametrize("hub", HUBS)
def test_cluster_hubs(N, O, hub):
    g = hub_graph(5000, hub, hub)
    for unit in (True, False):
        if not unit:
            weighted(g, hub)
        kn_o, kn_p = O.knobs(g, 2, 0.03, 1, 1), N.derive_knobs(g["n"], g["vwgt"], 2, 0.03, 1, 1)
        assert np.array_equal(O.lp_cluster(g, kn_o, 0), N.lp_cluster(g, kn_p, 0))


@pytest.mark.parametrize("n,hub", [(3000, 0), (3000, 256), (3000, 257), (140000, 0), (140000, 256)])
@pytest.mark.parametrize("rounds", [1, 2, 3, 4, 5, 7, 8, 12])
def test_cluster_quiet_rounds(N, O, graphs, n, hub, rounds):
    """Around the first round that passes over vertices that cannot move, with
    and without a row too long for it, as a team and as launches."""
    g = hub_graph(n, hub, hub) if hub else graphs.rgg2d(n, seed=n)
    for unit in (True, False):
        if not unit:
            weighted(g, hub + 1)
        kn_o, kn_p = O.knobs(g, 4, 0.03, 3, 1), N.derive_knobs(g["n"], g["vwgt"], 4, 0.03, 3, 1)
        kn_o.lpc_rounds = kn_p.lpc_rounds = rounds
        for bound in (kn_p.cluster_bound, 9):  # 9: weights near the bound decide
            kn_o.cluster_bound = kn_p.cluster_bound = bound
            assert np.array_equal(O.lp_cluster(g, kn_o, 1), N.lp_cluster(g, kn_p, 1))


@pytest.mark.parametrize("hubs", [(2048, 2049), (2049,) * 5, (8192, 8193, 129, 2048), (30000, 9000, 2500)])
def test_cluster_giant_rows(N, O, hubs):
    """Rows listed from both ends: a block's smaller table, its larger one and
    the one in global memory."""
    n = 40000
    rng = np.random.default_rng(len(hubs))
    lo = [np.arange(n - 1)] + [np.full(h, c) for c, h in enumerate(hubs)]
    hi = [np.arange(1, n)] + [rng.choice(np.arange(len(hubs) + 1, n), h, False) for h in hubs]
    edges = np.unique(np.stack([np.concatenate(lo), np.concatenate(hi)], 1), axis=0)
    g = csr_from_edges(n, [tuple(map(int, e)) for e in edges])
    for unit in (True, False):
        if not unit:
            weighted(g, 7)
        kn_o, kn_p = O.knobs(g, 2, 0.03, 1, 1), N.derive_knobs(n, g["vwgt"], 2, 0.03, 1, 1)
        for level in (0, 2):
            assert np.array_equal(O.lp_cluster(g, kn_o, level), N.lp_cluster(g, kn_p, level))
        part = skewed(n, 1100, 5)  # no dense counters: the refinement's tables
        kn_o, kn_p = O.knobs(g, 1100, 0.03, 1, 0), N.derive_knobs(n, g["vwgt"], 1100, 0.03, 1, 0)
        assert np.array_equal(O.lp_refine(g, kn_o, part, kn_o.upper_bound, 0),
                              N.lp_refine(g, kn_p, part, kn_p.upper_bound, 0))


def test_cluster_unsorted_rows(N, O, graphs):
    """Rows in no order and a target listed twice: no singleton shortcut."""
    g = graphs.rgg2d(3000, seed=4)
    rng = np.random.default_rng(0)
    adj = g["adjncy"].copy()
    for v in range(g["n"]):
        rng.shuffle(adj[g["xadj"][v]:g["xadj"][v + 1]])
    h = dict(g, adjncy=adj)
    kn_o, kn_p = O.knobs(h, 8, 0.03, 1, 0), N.derive_knobs(h["n"], h["vwgt"], 8, 0.03, 1, 0)
    assert np.array_equal(O.lp_cluster(h, kn_o, 0), N.lp_cluster(h, kn_p, 0))


@pytest.mark.parametrize("where", ["first", "last", "middle", "hub", "end"])
@pytest.mark.parametrize("n", [40, 3000, 40000])
def test_one_unsorted_row(N, O, where, n):
    """The check of the rows' order finds a single exchanged pair in any place
    (a row's target listed twice would otherwise take the singleton shortcut)."""
    rng = np.random.default_rng(n)
    edges = {(v, v + 1) for v in range(n - 1)} | {(n // 2, int(u)) for u in rng.integers(0, n, n // 3) if u != n // 2}
    g = csr_from_edges(n, sorted({(min(e), max(e)) for e in edges}))
    x, adj, wgt = g["xadj"], g["adjncy"].copy(), g["adjwgt"].copy()
    v = {"first": 1, "last": n - 2, "middle": n // 3, "hub": n // 2, "end": n // 2}[where]
    e = x[v + 1] - 2 if where == "end" else x[v] + (x[v + 1] - x[v]) // 2 - 1
    adj[e + 1], wgt[e + 1] = adj[e], wgt[e] + 2  # the same target twice
    h = dict(g, adjncy=adj, adjwgt=wgt)
    kn_o, kn_p = O.knobs(h, 2, 0.03, 1, 0), N.derive_knobs(n, h["vwgt"], 2, 0.03, 1, 0)
    assert np.array_equal(O.lp_cluster(h, kn_o, 0), N.lp_cluster(h, kn_p, 0))
    bad = dict(g, adjncy=g["adjncy"].copy())
    bad["adjncy"][e] = n
    with pytest.raises(Exception):
        N.kaffpa_ex(bad["xadj"], bad["adjncy"], 2)


def test_teams_side_by_side(N, graphs):
    """Workers share the device: every result is the single call's."""
    gs = [graphs.rgg2d(20000 + 977 * i, seed=i) for i in range(6)] + [graphs.rmat(13, samples=4 << 13, seed=1)]
    cuts, parts, status, _ = N.kaffpa_batch(gs, [2, 8, 16, 64, 5, 3, 8], 0.03, 7, N.FAST, workers=7)
    assert (status >= 0).all()
    for g, k, cut, part in zip(gs, [2, 8, 16, 64, 5, 3, 8], cuts, parts):
        _, c, p = N.kaffpa_ex(g["xadj"], g["adjncy"], k, 0.03, 7, N.FAST, vwgt=g["vwgt"], adjwgt=g["adjwgt"])
        assert c == cut and np.array_equal(p, part)


@pytest.mark.parametrize("n,k", [(900, 2), (1200, 64), (1700, 3), (2600, 8), (6000, 64), (20000, 5)])
def test_initial_partition_gangs(N, O, graphs, n, k):
    """Tries by a block and by clusters of 2 to 16 blocks (from 16384 entries
    on), thread rows and warp rows, several components, unreached nodes."""
    rng = np.random.default_rng(n)
    perm = rng.permutation(2 * n)[:n]  # half a graph: some nodes isolated
    half = graphs.rgg2d(2 * n, seed=n, r_factor=0.9)
    keep = np.zeros(2 * n, bool)
    keep[perm] = True
    src = np.repeat(np.arange(2 * n), np.diff(half["xadj"]))
    sel = keep[src] & keep[half["adjncy"]] & (src < half["adjncy"])
    new = np.cumsum(keep) - 1
    sparse = csr_from_edges(n, list(zip(new[src[sel]].tolist(), new[half["adjncy"][sel]].tolist())))
    dense = graphs.rmat(max(8, int(np.log2(n)) - 2), samples=24 * n, seed=n)
    for g in (graphs.rgg3d(n, seed=n, r_factor=0.8), sparse, dense):
        g["vwgt"] = rng.integers(1, 9, g["n"]).astype(np.int32)
        for mode in (0, 1):
            kn_o, kn_p = O.knobs(g, k, 0.03, 5, mode), N.derive_knobs(g["n"], g["vwgt"], k, 0.03, 5, mode)
            assert np.array_equal(O.initial_partition_batched(g, kn_o), N.initial_partition_device(g, kn_p))


@pytest.mark.parametrize("n,hub", [(1, 0), (33, 0), (256, 0), (257, 0), (2049, 0), (4097, 0), (40001, 0), (160000, 0),
                                   (5000, 32), (5000, 33), (5000, 128), (5000, 1025)])
def test_match_sizes(N, O, graphs, n, hub):
    """Teams of every form, rows of every batch remainder, and the reuse of
    proposals over the rounds, for unit weights, weights and ratings with ties."""
    g = hub_graph(n, hub, hub) if hub else graphs.rgg2d(n, seed=n) if n > 33 else \
        csr_from_edges(n, [(i, i + 1) for i in range(n - 1)])
    for unit in (True, False):
        if not unit:
            weighted(g, n + hub)
        src = np.repeat(np.arange(n), np.diff(g["xadj"])).astype(np.int64)
        rating = ((src + g["adjncy"]) * 7919 % 13).astype(np.uint32)  # symmetric, many equal
        for rounds in (1, 2, 16):
            kn_o, kn_p = O.knobs(g, 2, 0.03, 9, 0), N.derive_knobs(n, g["vwgt"], 2, 0.03, 9, 0)
            kn_o.match_rounds = kn_p.match_rounds = rounds
            for rq in (None, rating):
                assert np.array_equal(O.hem_match(g, kn_o, 1, rq), N.hem_match(g, kn_p, 1, rq))
