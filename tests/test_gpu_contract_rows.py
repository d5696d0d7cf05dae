"""Contraction rows of every length class against the CPU oracle: the warp's
table (up to 128 targets, 8192 entries), the block's counters beyond it, their
further passes (more than 2^20 coarse nodes), and the matching path's sorts
(64, 1024 entries) -- with unit, repeated and zero weights.  Also the cut of a
graph whose long rows are walked in pieces.  Integer outputs: equality.
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


def same(a, b):
    (ga, ma), (gb, mb) = a, b
    assert np.array_equal(ma, mb) and ga["n"] == gb["n"] and ga["m"] == gb["m"]
    for key in ("xadj", "adjncy", "adjwgt", "vwgt"):
        assert np.array_equal(ga[key], gb[key]), key


def hubs_graph(n, degrees, seed, unit):
    """A ring, and node i joined to degrees[i] random nodes (CSR by numpy)."""
    rng = np.random.default_rng(seed)
    s = [np.arange(n), np.arange(1, n + 1) % n]
    src, dst = [s[0]], [s[1]]
    for i, d in enumerate(degrees):
        t = rng.choice(np.arange(len(degrees) + 2, n - 2), d, replace=False)
        src.append(np.full(d, i))
        dst.append(t)
    src, dst = np.concatenate(src).astype(np.int64), np.concatenate(dst).astype(np.int64)
    lo, hi = np.minimum(src, dst), np.maximum(src, dst)
    key = np.unique(lo * n + hi)
    lo, hi = key // n, key % n
    a, b = np.concatenate([lo, hi]), np.concatenate([hi, lo])
    order = np.lexsort((b, a))
    a, b = a[order], b[order]
    w = np.ones(len(a), np.int32) if unit else ((np.minimum(a, b) * 7 + np.maximum(a, b)) % 5).astype(np.int32)
    xadj = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))])
    from kahip_b200.graphs import from_csr
    return from_csr(xadj, b, w, (np.arange(n) % 3 + 1).astype(np.int32))


@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("per", [1, 3, 40])
def test_row_lengths(N, O, unit, per):
    """per fine nodes a coarse node: the emission (1) and the gather path."""
    degrees = [30, 31, 60, 62, 63, 120, 124, 125, 126, 127, 130, 254, 256, 300, 1020, 1021, 1022, 1023, 1500, 5000]
    g = hubs_graph(40000, degrees, per, unit)
    label = np.arange(g["n"], dtype=np.int32) // per * per
    same(O.contract(g, label), N.contract(g, label))


@pytest.mark.parametrize("unit", [True, False])
def test_many_entries_few_targets(N, O, graphs, unit):
    """Coarse nodes of more than 8192 member entries and few targets, and all
    nodes but a few in one cluster."""
    g = graphs.rgg2d(60000, seed=3)
    if not unit:
        src = np.repeat(np.arange(g["n"]), np.diff(g["xadj"])).astype(np.int64)
        g["adjwgt"] = ((np.minimum(src, g["adjncy"]) * 7 + np.maximum(src, g["adjncy"])) % 5).astype(np.int32)
    label = (np.arange(g["n"]) // 5000 * 5000).astype(np.int32)
    same(O.contract(g, label), N.contract(g, label))
    label = np.where(np.arange(g["n"]) % 97 == 0, np.arange(g["n"]), 1).astype(np.int32)
    same(O.contract(g, label), N.contract(g, label))


@pytest.mark.parametrize("n,per", [((1 << 20) + 12345, 1), (3 * ((1 << 20) + 777), 3)])
def test_more_coarse_nodes_than_a_pass(N, O, n, per):
    g = hubs_graph(n, [200, 1500, 3000, 20000], 5, per == 1)
    label = (np.arange(n) // per * per).astype(np.int32)
    same(O.contract(g, label), N.contract(g, label))


@pytest.mark.parametrize("unit", [True, False])
def test_cut_of_long_rows(N, O, unit):
    """Rows of 127 to 9000 entries: within, on and across piece borders."""
    g = hubs_graph(30000, [125, 126, 127, 128, 2046, 2047, 2048, 4096, 9000], 7, unit)
    for k in (2, 17, 13000):
        part = np.random.default_rng(k).integers(0, k, g["n"]).astype(np.int32)
        cut, bw = N.edge_cut(g, part, k)
        assert cut == O.edge_cut(g, part) and np.array_equal(bw, O.block_weights(g, part, k))
