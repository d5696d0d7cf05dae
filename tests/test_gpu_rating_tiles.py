"""The rating network's training kernels at the edges of their tiles (64 nodes
a tile, 32 entries a chunk of a row): the CUDA-core forward, the loss and the
gradient against PyTorch autograd of the fp32 restatement.

Tolerances as for the larger graphs (BF16 activations, other summation
orders): probabilities within 0.05 and 2e-3 on average, gradients within 2 %
in norm, the loss within 1 %.
"""
import numpy as np
import pytest

from conftest import csr_from_edges
from test_gpu_learned import random_params, torch_forward

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def N():
    from kahip_b200 import native
    assert native.device_count() > 0, "no CUDA device"
    return native


def graph(n, hub, seed):
    """A path with some chords, node 0 joined to `hub` nodes, weights 1-5."""
    rng = np.random.default_rng(seed)
    edges = {(v, v + 1) for v in range(n - 1)}
    edges |= {(0, v) for v in range(1, min(hub, n - 1) + 1)}
    for _ in range(n // 3):
        a, b = sorted(int(x) for x in rng.integers(0, n, 2))
        if a != b:
            edges.add((a, b))
    edges = sorted(edges)
    g = csr_from_edges(n, edges, weights=[1 + (a * 3 + b) % 5 for a, b in edges])
    g["vwgt"] = rng.integers(1, 7, n).astype(np.int32)
    return g


@pytest.mark.parametrize("n,hub", [(2, 1), (33, 31), (63, 32), (64, 33), (65, 1), (127, 64), (128, 65), (129, 96),
                                   (64 * 296 + 1, 97)])
def test_forward_and_gradient(N, n, hub):
    import torch
    g = graph(n, hub, n)
    P = random_params(n)
    prob, _ = N.rating_infer(g, P, use_tc=False)
    s, Pt = torch_forward(g, P, st=True)
    ref = torch.sigmoid(s).detach().numpy()
    assert np.abs(prob - ref).max() < 5e-2 and np.abs(prob - ref).mean() < 2e-3
    src = np.repeat(np.arange(n), np.diff(g["xadj"]))
    label = ((src + g["adjncy"]) % 3 == 0).astype(np.uint8)  # symmetric
    grad, loss = N.rating_grad(g, label, P)
    y = torch.from_numpy(label.astype(np.float32))
    cut = float(y.sum())
    pos = min(50.0, max(1.0, (len(label) - cut) / cut)) if cut > 0 else 1.0
    w = torch.where(y > 0, torch.full_like(y, pos), torch.ones_like(y)) / max(1.0, pos * cut + len(label) - cut)
    lt = (w * torch.nn.functional.binary_cross_entropy_with_logits(s, y, reduction="none")).sum()
    lt.backward()
    gt = Pt.grad.numpy()
    assert abs(loss - float(lt.detach())) <= 0.01 * max(float(lt.detach()), 1e-6)
    assert np.linalg.norm(grad - gt) <= 0.02 * np.linalg.norm(gt)


def test_no_edges(N):
    g = csr_from_edges(70, [])
    grad, loss = N.rating_grad(g, np.zeros(0, np.uint8), random_params(1))
    assert loss == 0.0 and not grad.any()


@pytest.mark.parametrize("n,hub", [(1, 0), (2, 1), (127, 3), (128, 126), (129, 128), (1100, 1024), (1100, 1025),
                                   (128 * 148 + 1, 40), (128 * 148 * 4 + 5, 1500)])
def test_tensor_core_forward(N, n, hub):
    """Part tiles, one to five tiles a CTA (three are gathered ahead), nodes
    without edges, rows at the limit of the separate sums."""
    import torch
    g = graph(n, hub, n + 1)
    pad = 5  # isolated nodes at the end
    g = dict(g, n=n + pad, xadj=np.concatenate([g["xadj"], np.full(pad, g["xadj"][-1], g["xadj"].dtype)]),
             vwgt=np.concatenate([g["vwgt"], np.arange(pad, dtype=np.int32)]))
    P = random_params(n + 7)
    prob, rating = N.rating_infer(g, P, use_tc=True)
    if g["m"] == 0:
        assert prob.size == 0
        return
    s, _ = torch_forward(g, P)
    ref = torch.sigmoid(s).detach().numpy()
    assert np.abs(prob - ref).max() < 5e-2 and np.abs(prob - ref).mean() < 2e-3
    q = np.clip(np.floor((1.0 - prob) * np.float32(16777216.0)), 0, 16777215)
    assert np.array_equal(rating, q.astype(np.uint32))
