"""Contraction of short rows at the edges of its tiers, and matching with round
counts around the batches they are enqueued in, against the oracle event by event."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from thegraphpartitioning_b200._abi import GP_TR_CONTRACT, GP_TR_MATCH
from helpers import compare_traces, to_np, weighted

pytestmark = pytest.mark.gpu


def _ring(n, steps):
    """Every vertex linked to the ids `steps` before and after it."""
    v = torch.arange(n)
    return graphs.csr_from_edges(v.repeat(len(steps)), torch.cat([(v + s) % n for s in steps]), n)[:2]


def _cases():
    # matched pairs' walks of 2 * degree entries: 16 / 18 and 32 / 34 (one thread, 16 or
    # 32 registers; a warp), with many shared neighbours and with few
    for deg in (8, 9, 16, 17):
        near = list(range(1, deg // 2 + 1)) + ([1500] if deg % 2 else [])   # n / 2: one entry
        yield f"near{deg}", _ring(3000, near), None, {}
        far = [1 + 37 * i for i in range(deg // 2)] + ([1500] if deg % 2 else [])
        yield f"far{deg}_w", _ring(3000, far), "w", {}
    for rounds in (1, 3, 4, 5, 8, 9):
        yield f"rounds{rounds}", graphs.rmat(12, seed=2)[:2], None, {"match_rounds": rounds}
        yield f"rounds{rounds}_nohop_w", graphs.grid2d(70, 60), "w", {"match_rounds": rounds, "two_hop": -1}
    yield "isolated", graphs.csr_from_edges(torch.arange(0, 4000, 2), torch.arange(0, 4000, 2) ^ 6, 4000)[:2], None, {}


CASES = list(_cases())


@pytest.mark.parametrize("name,g,w,opts", CASES, ids=[c[0] for c in CASES])
def test_coarsening_matches_oracle(oracle_mod, gp, cuda, name, g, w, opts):
    rp, ci = to_np(*g)
    ew, vw = weighted(rp, ci, seed=5) if w else (None, None)
    opts = dict(opts, coarsen_to=64, init_trials=2, refine_max_iters=1)
    kinds = (GP_TR_MATCH, GP_TR_CONTRACT)
    _, s_ref, ev = oracle_mod.partition(rp, ci, 2, 0.2, 4, vwgt=vw, ewgt=ew, options=opts, trace=True)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    _, s_gpu, ev_gpu = gp.partition(d(rp), d(ci), 2, 0.2, 4, vwgt=d(vw), ewgt=d(ew), options=opts, trace=set(kinds))
    compare_traces([e for e in ev if e["kind"] in kinds], ev_gpu)
    assert s_ref["levels"] == s_gpu["levels"]
