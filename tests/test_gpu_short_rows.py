"""Rows around the bucket edges (16 / 17 and 32 / 33 entries) and levels around
the sizes from which short rows get their own launches, against the oracle
event by event."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from helpers import compare_traces, to_np, weighted

pytestmark = pytest.mark.gpu


def _circulant(n, deg):
    """Every vertex linked to its deg / 2 next and previous ids: rows of exactly deg entries (deg even)."""
    v = torch.arange(n)
    return graphs.csr_from_edges(v.repeat(deg // 2), torch.cat([(v + d) % n for d in range(1, deg // 2 + 1)]), n)[:2]


def _mixed(n, seed=0):
    """Rows of 1..40 entries side by side, the lengths changing from row to row."""
    v = torch.arange(n)
    s, d = [], []
    for j in range(1, 21):
        keep = (graphs.mix64(v * 31 + seed) & 31) >= j
        s.append(v[keep])
        d.append((v[keep] + j) % n)
    return graphs.csr_from_edges(torch.cat(s), torch.cat(d), n)[:2]


def _cases():
    for deg in (8, 16, 18, 32, 34):
        yield f"circulant{deg}", _circulant(1500, deg), 7, None
    # either side of the sizes from which short rows are launched apart
    # (24,576 for the matching, 32,768 for the connectivity pass)
    yield "rows24575", _circulant(24575, 4), 3, None
    yield "rows24576_w", _circulant(24576, 16), 3, "w"
    yield "rows32767", _circulant(32767, 10), 300, None
    yield "rows32768", _circulant(32768, 16), 300, None
    yield "mixed40k_w", _mixed(40000), 12, "w"
    yield "mixed2k", _mixed(2000, 5), 5, None
    # appends of four rows per thread (262,144 rows and more)
    yield "grid513_k4", graphs.grid2d(513, 513), 4, None


CASES = list(_cases())


@pytest.mark.parametrize("name,g,k,w", CASES, ids=[c[0] for c in CASES])
def test_short_rows_match_oracle(oracle_mod, gp, cuda, name, g, k, w):
    rp, ci = to_np(*g)
    ew, vw = weighted(rp, ci, seed=2) if w else (None, None)
    opts = {"init_trials": 4}
    p_ref, _, ev_ref = oracle_mod.partition(rp, ci, k, 0.03, 3, vwgt=vw, ewgt=ew, options=opts, trace=True)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    p_gpu, _, ev_gpu = gp.partition(d(rp), d(ci), k, 0.03, 3, vwgt=d(vw), ewgt=d(ew), options=opts, trace=True)
    compare_traces(ev_ref, ev_gpu)
    # without the trace the proposals are not stored apart
    p2, _, _ = gp.partition(d(rp), d(ci), k, 0.03, 3, vwgt=d(vw), ewgt=d(ew), options=opts)
    assert np.array_equal(p_ref, p_gpu.cpu().numpy()) and np.array_equal(p_ref, p2.cpu().numpy())
