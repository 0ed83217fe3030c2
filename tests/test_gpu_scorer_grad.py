"""The scorer's gradient at the sizes where its kernels change: rows of 16 / 17 /
32 / 33 entries and a hub, vertex counts around the 64-vertex chunks of the weight
gradients, against the float64 chain rule with the bounds its other tests use."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from helpers import to_np, weighted

pytestmark = pytest.mark.gpu


def _ring(n, deg):
    v = torch.arange(n)
    return graphs.csr_from_edges(v.repeat(deg // 2), torch.cat([(v + s) % n for s in range(1, deg // 2 + 1)]), n)[:2]


def _mixed(n):
    """Rows of 16, 17, 32, 33 entries and two hubs of several hundred."""
    v = torch.arange(n)
    a = [v.repeat(8), torch.arange(0, n, 3), torch.zeros(n // 2, dtype=torch.int64), torch.full((n // 3,), 5)]
    b = [torch.cat([(v + s) % n for s in range(1, 9)]), (torch.arange(0, n, 3) + n // 2) % n,
         torch.arange(20, 20 + n // 2), torch.arange(40, 40 + n // 3)]
    return graphs.csr_from_edges(torch.cat(a), torch.cat(b), n)[:2]


CASES = [("n3", _ring(3, 2), None), ("n63_d16", _ring(63, 16), "w"), ("n64_d18", _ring(64, 18), None),
         ("n65_d32", _ring(65, 32), "w"), ("n129_d34", _ring(129, 34), None), ("mixed", _mixed(1201), "w"),
         ("rmat", graphs.rmat(12, seed=9)[:2], None)]


@pytest.mark.parametrize("name,g,w", CASES, ids=[c[0] for c in CASES])
def test_gradient_at_row_edges(gp, cuda, name, g, w):
    from oracle import gnn_ref
    rp, ci = to_np(*g)
    ew, vw = weighted(rp, ci, seed=3) if w else (None, None)
    p = gnn_ref.init_params(5)
    p[gnn_ref.O_GAMMA], p[gnn_ref.O_DELTA], p[gnn_ref.O_ETA] = 0.3, 0.1, 0.2
    n = len(rp) - 1
    part = (np.arange(n) * 3 // n).astype(np.int32)
    src = np.repeat(np.arange(n), np.diff(rp))
    label = (part[src] == part[ci]).astype(np.uint8)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    loss, grad = gp.GNN(p).grad(d(rp), d(ci), d(label), d(vw), d(ew), 1)
    loss_ref, ref = gnn_ref.loss_and_grad(gnn_ref.bf16_round(p), rp, ci, label, vw, ew, 1)
    assert abs(loss - loss_ref) <= 1e-5 + 1e-5 * abs(loss_ref)
    cut = [gnn_ref.O_W1, gnn_ref.O_B1, gnn_ref.O_P, gnn_ref.O_W2, gnn_ref.O_B2, gnn_ref.O_Z, gnn_ref.O_A, gnn_ref.NPARAM]
    for lo, hi in zip(cut, cut[1:]):
        rel = np.linalg.norm(grad[lo:hi] - ref[lo:hi]) / max(np.linalg.norm(ref[lo:hi]), 1e-12)
        assert rel < 2e-3, (name, lo, rel)
