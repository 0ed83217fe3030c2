"""Cuts of the initial partition's trials, added up for 16 trials at a time: trial
counts around 16, labels of 8 and 16 bits, sizes at which the labels no longer fit
on chip, weights; the kept trial and its labels against the oracle."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from thegraphpartitioning_b200._abi import GP_TR_INITPART
from helpers import compare_traces, to_np, weighted

pytestmark = pytest.mark.gpu

CASES = [(1200, 60, 6, None, 1), (1200, 60, 6, "w", 15), (1200, 60, 6, None, 16), (1201, 60, 7, "w", 17),
         (1500, 50, 256, None, 33), (1500, 50, 257, "w", 20), (1500, 50, 300, None, 48),
         (15, 14, 3, None, 5), (5000, 16, 4, "w", 18),
         (7100, 12, 260, None, 3), (7200, 12, 260, None, 3), (14000, 8, 5, None, 3), (14400, 8, 5, "w", 3)]


@pytest.mark.parametrize("n,deg,k,w,trials", CASES)
def test_kept_trial_matches_oracle(oracle_mod, gp, cuda, n, deg, k, w, trials):
    rp, ci = to_np(*graphs.erdos_renyi(n, float(deg), seed=n + k))
    ew, vw = weighted(rp, ci, seed=4) if w else (None, None)
    opts = {"coarsen_to": n, "init_trials": trials, "refine_max_iters": 1}
    _, _, ev = oracle_mod.partition(rp, ci, k, 0.1, 3, vwgt=vw, ewgt=ew, options=opts, trace=True)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    _, _, ev_gpu = gp.partition(d(rp), d(ci), k, 0.1, 3, vwgt=d(vw), ewgt=d(ew), options=opts, trace={GP_TR_INITPART})
    compare_traces([e for e in ev if e["kind"] == GP_TR_INITPART], ev_gpu)
