"""Levels of more than 4 M entries with long rows: the pass that ends a level (the
last iteration, or the last one patience allows) takes the cut from the moved rows
alone; iterations, kept states and cuts against the oracle."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from helpers import compare_traces, to_np, weighted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,iters,patience,imb,w", [(64, 1, 4, 0.03, None), (64, 2, 1, 0.03, "w"), (8, 6, 1, 0.3, None),
                                                    (300, 4, 2, 0.05, None), (64, 9, 3, 0.01, None)])
def test_last_pass_matches_oracle(oracle_mod, gp, cuda, k, iters, patience, imb, w):
    rp, ci = to_np(*graphs.rmat(18, seed=6)[:2])
    assert len(ci) > 1 << 22
    ew, vw = weighted(rp, ci, seed=2) if w else (None, None)
    opts = {"init_trials": 2, "coarsen_to": 60000, "refine_max_iters": iters, "refine_patience": patience}
    p_ref, s_ref, ev_ref = oracle_mod.partition(rp, ci, k, imb, 8, vwgt=vw, ewgt=ew, options=opts, trace=True)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    _, _, ev_gpu = gp.partition(d(rp), d(ci), k, imb, 8, vwgt=d(vw), ewgt=d(ew), options=opts, trace=True)
    compare_traces(ev_ref, ev_gpu)
    part, s, _ = gp.partition(d(rp), d(ci), k, imb, 8, vwgt=d(vw), ewgt=d(ew), options=opts)
    assert np.array_equal(p_ref, part.cpu().numpy()) and s["cut"] == s_ref["cut"]
