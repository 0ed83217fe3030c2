"""The loss's sum in 64 bits: with every scorer parameter but the constant zero, each
entry's float32 term depends on its label alone, so the mean over a large graph is
known to the last bit from the two terms."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["grid3d", "rmat"])
def test_loss_of_constant_logits(gp, cuda, family):
    from oracle import gnn_ref
    p = np.zeros(gnn_ref.NPARAM, np.float32)
    p[gnn_ref.O_DELTA] = 0.37
    m = gp.GNN(p)
    pair = [torch.tensor(x, device=cuda) for x in ([0, 1, 2], [1, 0])]
    pair[0], pair[1] = pair[0].long(), pair[1].int()
    term = [m.grad(pair[0], pair[1], torch.full((2,), y, dtype=torch.uint8, device=cuda))[0] for y in (0, 1)]
    t = float(torch.tensor(0.37).bfloat16())
    for y in (0, 1):   # the terms themselves: expf and log1pf within 2 ulp each
        assert abs(term[y] - (max(t, 0) - t * y + np.log1p(np.exp(-abs(t))))) <= 5 * 2.0 ** -23
    g = graphs.grid3d(101, 97, 89) if family == "grid3d" else graphs.rmat(17, seed=2)[:2]
    rp, ci = g[0].to(cuda), g[1].to(cuda)
    label = (torch.arange(ci.numel(), device=cuda) * 2654435761 % 7 < 3).to(torch.uint8)
    loss = m.grad(rp, ci, label)[0]
    ones = int(label.sum())
    want = (term[1] * ones + term[0] * (ci.numel() - ones)) / ci.numel()
    # one rounding to float32 (half an ulp: 2^-24 relative), the sum of 64-bit terms below it
    assert abs(loss - want) <= want * (2.0 ** -24 + 1e-12)
