"""The calls this library's speed is judged by: whole partitionings through
the public entry points (host buffers, device buffers, batches, populations,
evolution), and the learned edge rating's forward and backward passes.

`listed()` names the fixed cases, `draw(rng)` gives another one of the same
ranges, `prepare` builds what a caller holds before the call, `run` is the
call, `work` the bytes and operations it cannot do without, and `exact` the
64-bit values of the floating-point outputs.

Graphs are the library's seeded generators: random geometric graphs in two
and three dimensions (meshes), 5-point grids and R-MAT (social networks).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from kahip_b200 import graphs, learned, native

MODES = {"fast": native.FAST, "eco": native.ECO, "fastsocial": native.FASTSOCIAL}


def listed() -> list:
    return [
        # the smallest call in use: a mesh of a thousand nodes halved through
        # the host interface, where launches and synchronisations are all
        {"name": "host_grid_1k_k2", "kind": "host", "graph": "grid", "n": 1023, "k": 2, "eps": 0.03,
         "mode": "fast", "weighted": False},
        # the interface's everyday call: a mid-size mesh, 8 blocks
        {"name": "host_rgg2d_32k_k8", "kind": "host", "graph": "rgg2d", "n": 32768, "k": 8, "eps": 0.03,
         "mode": "fast", "weighted": False},
        # a weighted finite-element-like mesh (node and edge weights), the
        # quality preset, a ragged size and a block count off the powers of two
        {"name": "host_rgg3d_200k_eco_wgt", "kind": "host", "graph": "rgg3d", "n": 200003, "k": 27, "eps": 0.03,
         "mode": "eco", "weighted": True},
        # the benchmark configuration: the largest single graph, device-resident
        {"name": "dev_rgg2d_16m_k64", "kind": "device", "graph": "rgg2d", "n": 1 << 24, "k": 64, "eps": 0.03,
         "mode": "fast", "weighted": False},
        # the quality preset on a large mesh (Jet refinement), odd size
        {"name": "dev_rgg2d_4m_eco_k64", "kind": "device", "graph": "rgg2d", "n": 4000037, "k": 64, "eps": 0.03,
         "mode": "eco", "weighted": False},
        # many blocks on a 3D mesh: the initial partitioning's share is largest
        {"name": "dev_rgg3d_3m_k256", "kind": "device", "graph": "rgg3d", "n": 3000017, "k": 256, "eps": 0.03,
         "mode": "fast", "weighted": False},
        # a social network: skewed degrees, weighted edges, dense coarse graphs
        {"name": "dev_rmat_1m_k64", "kind": "device", "graph": "rmat", "n": 1 << 20, "k": 64, "eps": 0.03,
         "mode": "fastsocial", "weighted": False},
        # matching coarsening on the shipped learned rating
        {"name": "dev_rgg2d_1m_learned_k32", "kind": "learned", "graph": "rgg2d", "n": 1000003, "k": 32, "eps": 0.03,
         "mode": "fast", "weighted": False},
        # many independent graphs of uneven size in one call
        {"name": "batch_96", "kind": "batch", "count": 96, "nmin": 1000, "nmax": 200000, "eps": 0.03},
        # many seeds of one device-resident graph
        {"name": "population_16_256k_k16", "kind": "population", "graph": "rgg2d", "n": 262147, "k": 16, "eps": 0.03,
         "mode": "fast", "weighted": False, "count": 16},
        # an evolutionary search: population, then rounds of combines
        {"name": "evolve_128k_k8", "kind": "evolve", "graph": "rgg2d", "n": 131071, "k": 8, "eps": 0.03,
         "mode": "fast", "weighted": False, "population": 4, "generations": 2, "per_generation": 2},
        # one training step of the edge rating: loss and gradient of one graph
        {"name": "rating_grad_32k", "kind": "grad", "graph": "rgg2d", "n": 32771, "k": 16, "weighted": True},
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["host", "host", "device", "device", "device", "learned", "batch", "population", "evolve", "grad",
                       "infer"])
    eps = rng.choice([0.01, 0.03, 0.03, 0.05])
    k = rng.choice([2, 3, 5, 8, 16, 27, 32, 64, 100, 128, 256])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(8, 90), "nmin": 1000, "nmax": _log_int(rng, 4000, 200000), "eps": eps}
    if kind == "infer":  # one probability per entry: a mesh whose entries number the same for every seed
        return {"kind": kind, "graph": "grid", "n": _log_int(rng, 2000, 250000), "k": 16, "weighted": True}
    if kind == "grad":
        return {"kind": kind, "graph": rng.choice(["rgg2d", "rgg3d"]), "n": _log_int(rng, 2000, 32000),
                "k": rng.choice([4, 16, 64]), "weighted": rng.random() < 0.5}
    graph = rng.choice(["rgg2d", "rgg2d", "rgg3d", "grid", "rmat"])
    case = {"kind": kind, "graph": graph, "k": k, "eps": eps, "mode": rng.choice(["fast", "fast", "eco"]),
            "weighted": rng.random() < 0.3}
    if kind == "host":
        n = _log_int(rng, 1000, 250000)
    elif kind == "device":
        n = _log_int(rng, 30000, 4000000 if case["mode"] == "eco" or k <= 8 else 15000000)
    elif kind == "learned":
        n = _log_int(rng, 30000, 900000)
        case["graph"] = graph = "rgg2d" if graph == "rmat" else graph
    elif kind == "population":
        n = _log_int(rng, 10000, 200000)
        case["count"] = rng.randint(3, 12)
    else:
        n = _log_int(rng, 10000, 100000)
        case.update(population=rng.randint(2, 4), generations=rng.randint(1, 2), per_generation=rng.randint(1, 2))
    if graph == "rmat":  # its sizes are powers of two, and its passes the costliest
        n = 1 << max(10, min(int(math.log2(n)), 19 if kind in ("host", "device") else 14))
    case["n"] = n
    return case


# ------------------------------------------------------------------ inputs

def _grid_side(n) -> int:
    return max(2, int(math.sqrt(n)))


def _graph(case, seed) -> dict:
    n = case["n"]
    if case["graph"] == "grid":
        nx = _grid_side(n)
        g = graphs.grid2d(nx, n // nx)
    elif case["graph"] == "rgg2d":
        g = graphs.rgg2d(n, seed=seed)
    elif case["graph"] == "rgg3d":
        g = graphs.rgg3d(n, seed=seed)
    else:
        g = graphs.rmat(int(math.log2(n)), seed=seed)
    if case["weighted"]:
        rng = np.random.default_rng(seed)
        g["vwgt"] = rng.integers(1, 6, g["n"], dtype=np.int32)
        # a weight per undirected edge, the same in both directions
        src = np.repeat(np.arange(g["n"], dtype=np.int64), np.diff(g["xadj"]))
        lo, hi = np.minimum(src, g["adjncy"]), np.maximum(src, g["adjncy"])
        h = (lo * 1000003 + hi * 7919 + seed) * 2654435761 & 0xFFFFFFFF
        g["adjwgt"] = (1 + (h >> 16) % 9).astype(np.int32)
    return g


def _on_gpu(g) -> dict:
    d = {key: torch.from_numpy(g[key]).cuda() for key in ("xadj", "adjncy", "adjwgt", "vwgt")}
    d["n"] = g["n"]
    return d


def _params():
    return learned.load_model()[0]


def prepare(case, seed) -> dict:
    kind = case["kind"]
    st = {"case": case, "seed": seed & 0xFFFF}
    if kind == "batch":
        # the mix of kinds, sizes and block counts is the case's, the graphs are the seed's
        specs = graphs.batch_specs(case["count"], case["count"], case["nmin"], case["nmax"])
        st["items"] = [(graphs.batch_graph((gk, n, k, gs ^ seed)), k) for gk, n, k, gs in specs]
        return st
    g = _graph(case, seed)
    if kind in ("host", "evolve", "grad", "infer"):
        if not case["weighted"] and kind == "host":
            g["vwgt"] = g["adjwgt"] = None  # unit weights, as the interface takes them
        st["g"] = g
    else:
        st["g"] = _on_gpu(g)
        st["part"] = torch.empty(case.get("count", 1) * g["n"], dtype=torch.int32, device="cuda")
    if kind in ("learned", "evolve"):
        kn = native.derive_knobs(g["n"], g["vwgt"], case["k"], case["eps"], st["seed"], MODES[case["mode"]])
        if kind == "learned":
            st["model"] = _params()
            kn.coarsening = 2
            kn.rating_model = st["model"].ctypes.data
        st["knobs"] = kn
    if kind in ("grad", "infer"):
        st["model"] = _params()
        # an edge is cut when its ends fall into different id ranges (ids
        # follow the geometry, so the ranges are strips of the domain)
        block = np.arange(g["n"], dtype=np.int64) * case["k"] // g["n"]
        st["label"] = (np.repeat(block, np.diff(g["xadj"])) != block[g["adjncy"]]).astype(np.uint8)
    return st


def run(st):
    case, g = st["case"], st.get("g")
    kind = case["kind"]
    if kind == "host":
        _, cut, part = native.kaffpa_ex(g["xadj"], g["adjncy"], case["k"], case["eps"], st["seed"],
                                        MODES[case["mode"]], vwgt=g["vwgt"], adjwgt=g["adjwgt"])
        return cut, part
    if kind == "device":
        _, cut = native.kaffpa_device(g["n"], g["xadj"], g["adjncy"], g["adjwgt"], g["vwgt"], st["part"], case["k"],
                                      case["eps"], st["seed"], MODES[case["mode"]])
        return cut, st["part"]
    if kind == "learned":
        _, cut = native.kaffpa_device_knobs(g["n"], g["xadj"], g["adjncy"], g["adjwgt"], g["vwgt"], st["part"],
                                            st["knobs"])
        return cut, st["part"]
    if kind == "batch":
        cuts, parts, _, _ = native.kaffpa_batch([x for x, _ in st["items"]], [k for _, k in st["items"]], case["eps"],
                                                st["seed"], native.FAST)
        return cuts, np.concatenate(parts)
    if kind == "population":
        seeds = np.arange(st["seed"], st["seed"] + case["count"], dtype=np.int32)
        cuts, _ = native.kaffpa_population(g["n"], g["xadj"], g["adjncy"], g["adjwgt"], g["vwgt"], st["part"],
                                           case["k"], seeds, case["eps"], MODES[case["mode"]])
        return cuts, st["part"]
    if kind == "evolve":
        _, cut, part, history = native.kaffpae(g, st["knobs"], case["population"], case["generations"],
                                               case["per_generation"])
        return cut, part, history
    if kind == "infer":
        return native.rating_infer(g, st["model"])
    grad, loss = native.rating_grad(g, st["label"], st["model"])
    return grad, loss


# -------------------------------------------------------------------- work

def _entries(graph, n) -> float:
    """Directed entries the generators give on average (edges of the domain
    cut off a few per cent)."""
    if graph == "grid":
        return 4.0 * n
    if graph == "rgg2d":
        return n * math.pi * 0.55 ** 2 * math.log(n) * 0.99
    if graph == "rgg3d":
        return n * 4.0 / 3.0 * math.pi * 0.55 ** 3 * math.log(n) * 0.97
    return 29.0 * n


def work(case) -> dict:
    kind = case["kind"]
    if kind == "batch":
        b = 0.0
        for gk, n, _, _ in graphs.batch_specs(case["count"], case["count"], case["nmin"], case["nmax"]):
            m = _entries("rgg2d", n) if gk == 0 else 4.0 * n if gk == 1 else 7.0 * n
            b += 16.0 * n + 8.0 * m
        return {"bytes": b, "flops": 0}
    n, m = case["n"], _entries(case["graph"], case["n"])
    # CSR in (weights where the call passes them), block ids out
    weights = kind != "host" or case["weighted"]
    b = 4.0 * (n + 1) + 4.0 * m + (4.0 * n + 4.0 * m if weights else 0.0)
    # operations of the rating network: three layers on [h | mean h], the
    # aggregation, the edge head
    net = n * (2.0 * (2 * 64 + 3 * 128 * 64 + 64 * 32)) + m * (3 * 2 * 64 + 32 * 7.0)
    if kind == "grad":
        return {"bytes": b + m + 8.0 * native.RATING_PARAMS, "flops": 3.0 * net}
    if kind == "infer":
        return {"bytes": b + 8.0 * m + 4.0 * native.RATING_PARAMS, "flops": net}
    return {"bytes": b + 4.0 * n * case.get("count", 1), "flops": net if kind == "learned" else 0}


# ------------------------------------------------------------------- exact

def _network(g, model):
    """The rating network in 64 bits on BF16 weights (activations are not
    rounded): logits per directed entry and the parameter vector."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = torch.float64
    n, Hd, Z = g["n"], 64, 32
    deg = torch.from_numpy(np.diff(g["xadj"]).astype(np.int64)).to(dev)
    adj = torch.from_numpy(g["adjncy"].astype(np.int64)).to(dev)
    w = torch.from_numpy(g["adjwgt"].astype(np.float64)).to(dev)
    vw = torch.from_numpy(g["vwgt"].astype(np.int64)).to(dev)
    src = torch.repeat_interleave(torch.arange(n, device=dev), deg)
    P = torch.from_numpy(model).to(torch.bfloat16).to(f64).to(dev).requires_grad_(True)
    at = 0

    def take(*shape):
        nonlocal at
        size = math.prod(shape)
        at += size
        return P[at - size:at].view(*shape)

    W0, b0 = take(Hd, 2), take(Hd)
    layers = [(take(Hd, 2 * Hd), take(Hd)) for _ in range(3)]
    Wz, bz, Wf, wo, bo = take(Z, Hd), take(Z), take(Z, 2), take(Z), take(1)
    x = torch.stack([torch.log2(1 + deg.to(f64)) / 8, torch.log2(vw.clamp(min=1).to(f64)) / 8], 1)
    h = torch.relu(x @ W0.T + b0)
    wd = torch.zeros(n, dtype=f64, device=dev).index_add_(0, src, w)
    inv = torch.where(wd > 0, 1 / wd.clamp(min=1e-30), torch.zeros_like(wd))
    for W, b in layers:
        mean = torch.zeros(n, Hd, dtype=f64, device=dev).index_add(0, src, w[:, None] * h[adj]) * inv[:, None]
        h = torch.relu(torch.cat([h, mean], 1) @ W.T + b)
    z = h @ Wz.T + bz
    f0 = torch.log2(w.clamp(min=1)) / 8
    f1 = torch.log2(1 + w * w / (vw[src] * vw[adj]).to(f64)) / 8
    t = z[src] + z[adj] + f0[:, None] * Wf[:, 0] + f1[:, None] * Wf[:, 1]
    return torch.relu(t) @ wo + bo, P


def exact(case, seed):
    if case["kind"] not in ("grad", "infer"):
        return None
    st = prepare(case, seed)
    s, P = _network(st["g"], st["model"])
    if case["kind"] == "infer":
        return torch.sigmoid(s).detach().cpu().numpy(), None
    y = torch.from_numpy(st["label"]).to(s.device).to(torch.float64)
    cut = float(y.sum())
    pos = min(50.0, max(1.0, (len(y) - cut) / cut)) if cut > 0 else 1.0
    wt = torch.where(y > 0, torch.full_like(y, pos), torch.ones_like(y)) / max(1.0, pos * cut + len(y) - cut)
    loss = (wt * torch.nn.functional.binary_cross_entropy_with_logits(s, y, reduction="none")).sum()
    loss.backward()
    return P.grad.cpu().numpy(), float(loss.detach())
