"""Long rows with neighbouring ids: the scorer's logits against the float64
reference, and its time, which depends on the rows and not on how they are numbered."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from helpers import to_np

pytestmark = pytest.mark.gpu


def _hubs(n, nhub, deg, stride, seed=0):
    """nhub vertices of about deg entries at ids 0, stride, 2 stride, ..., among n that else have two."""
    g = torch.Generator().manual_seed(seed)
    hub = torch.arange(nhub) * stride
    src = hub.repeat_interleave(deg)
    dst = torch.randint(0, n, (src.numel(),), generator=g)
    v = torch.arange(n)
    keep = src != dst
    return graphs.csr_from_edges(torch.cat([src[keep], v]), torch.cat([dst[keep], (v + 1) % n]), n)[:2]


@pytest.mark.parametrize("n,nhub,deg,stride", [(65, 33, 31, 1), (900, 64, 40, 1), (4000, 40, 300, 3), (9001, 33, 2600, 1),
                                               (9001, 5, 5000, 31)])
def test_scores_of_neighbouring_hubs(gp, cuda, n, nhub, deg, stride):
    from oracle import gnn_ref
    rp, ci = to_np(*_hubs(n, nhub, deg, stride))
    p = gnn_ref.init_params(4)
    p[gnn_ref.O_GAMMA], p[gnn_ref.O_DELTA], p[gnn_ref.O_ETA] = 0.3, 0.1, 0.9
    want = gnn_ref.forward(gnn_ref.bf16_round(p), rp, ci, None, None, level=1)
    _, logit = gp.GNN(p).forward(torch.from_numpy(rp).to(cuda), torch.from_numpy(ci).to(cuda), level=1)
    # the bound the scorer's other numerics tests use: 2e-4 absolute + relative
    assert np.all(np.abs(logit.cpu().numpy() - want) <= 2e-4 + 2e-4 * np.abs(want))


def test_time_does_not_depend_on_the_numbering(gp, cuda):
    """32 rows of 100,000 entries side by side against the same rows far apart: one
    warp sweeping all of the former took eight times as long."""
    m, times = gp.default_gnn(), []
    for stride in (1, 6000):
        rp, ci = (x.to(cuda) for x in _hubs(200000, 32, 100000, stride))
        m.forward(rp, ci)
        ev = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(); m.forward(rp, ci); b.record(); torch.cuda.synchronize()
            ev.append(a.elapsed_time(b))
        times.append(sorted(ev)[3])
    assert times[0] < 2 * times[1], times
