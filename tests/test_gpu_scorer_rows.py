"""The scorer at the sizes where its kernels change: rows of 8 / 9 / 16 / 17
entries, the row counts from which short rows take their own launch (24,576) and
the layers two vertices per thread (131,072), against the float64 reference."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from helpers import to_np, weighted

pytestmark = pytest.mark.gpu


def _ring(n, deg):
    v = torch.arange(n)
    return graphs.csr_from_edges(v.repeat(deg // 2), torch.cat([(v + s) % n for s in range(1, deg // 2 + 1)]), n)[:2]


def _cases():
    yield "n33_d2", _ring(33, 2), None
    yield "d8", _ring(24575, 8), None
    yield "d10_w", _ring(24576, 10), "w"
    yield "d16", _ring(24601, 16), None
    yield "d18_w", _ring(3001, 18), "w"
    yield "d34", _ring(2000, 34), None
    yield "wide", _ring(131071, 4), None
    yield "wide2_w", _ring(131072 + 37, 6), "w"
    yield "rmat", graphs.rmat(15, seed=4)[:2], None


CASES = list(_cases())


@pytest.mark.parametrize("name,g,w", CASES, ids=[c[0] for c in CASES])
def test_scores_match_reference(gp, cuda, name, g, w):
    from oracle import gnn_ref
    rp, ci = to_np(*g)
    ew, vw = weighted(rp, ci, seed=7) if w else (None, None)
    p = gnn_ref.init_params(3)
    p[gnn_ref.O_GAMMA], p[gnn_ref.O_DELTA], p[gnn_ref.O_ETA] = 0.3, 0.1, 0.2
    want = gnn_ref.forward(gnn_ref.bf16_round(p), rp, ci, vw, ew, level=1)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    m = gp.GNN(p)
    prio, logit = m.forward(d(rp), d(ci), d(vw), d(ew), level=1)
    logit = logit.cpu().numpy().astype(np.float64)
    # the bound the scorer's other numerics tests use: 2e-4 absolute + relative
    assert np.all(np.abs(logit - want) <= 2e-4 + 2e-4 * np.abs(want))
    # priorities are the rounded float32 logits
    q = np.rint(logit.astype(np.float32) * np.float32(65536.0)).clip(-2.0 ** 30, 1073741696.0)
    assert np.array_equal(prio.cpu().numpy(), (q.astype(np.int64) + (1 << 30)).astype(np.int32))
    # the same bits on every run
    prio2, logit2 = m.forward(d(rp), d(ci), d(vw), d(ew), level=1)
    assert torch.equal(prio, prio2)
