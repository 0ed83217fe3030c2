"""Rebalancing steps around the sizes where their path changes, scans and sorts
around theirs, against the oracle event by event."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from helpers import compare_traces, to_np, weighted

pytestmark = pytest.mark.gpu


def _cases():
    # k = 2 at exact balance: half the vertices are candidates of the first rebalance
    # step: one block up to 4,096 candidates, the whole chip above, on levels below
    # and above 16,384 vertices
    for n in (8000, 8400, 16384, 16500, 33000):
        yield f"rgg{n}_k2", graphs.random_geometric(n, 8.0, seed=n), 2, 0.0, None, {"coarsen_to": n}
    yield "rgg20k_k2_w", graphs.random_geometric(20000, 8.0, seed=4), 2, 0.0, "w", {"coarsen_to": 5000}
    # more than 256 parts: three sort passes (the result is copied back), 16-bit part ids
    yield "er40k_k300_w", graphs.erdos_renyi(40000, 8.0, seed=5), 300, 0.01, "w", {}
    yield "chunglu_k1024", graphs.chung_lu(60000, 200000, seed=6), 1024, 0.02, None, {}
    # collected one vertex per thread and 32 per thread (1,048,576 vertices on)
    yield "grid1023_k2", graphs.grid2d(1023, 1025), 2, 0.0, None, {"refine_max_iters": 3}
    yield "grid1024_k2", graphs.grid2d(1024, 1024), 2, 0.0, None, {"refine_max_iters": 3}
    yield "grid1025_k260", graphs.grid2d(1025, 1027), 260, 0.0, None, {"refine_max_iters": 3}
    # more iterations than the ring of status blocks holds
    yield "grid_patience100", graphs.grid2d(150, 120), 3, 0.0, None, {"refine_patience": 100, "refine_max_iters": 150}


CASES = list(_cases())


@pytest.mark.parametrize("name,g,k,imb,w,opts", CASES, ids=[c[0] for c in CASES])
def test_rebalance_matches_oracle(oracle_mod, gp, cuda, name, g, k, imb, w, opts):
    rp, ci = to_np(*g)
    ew, vw = weighted(rp, ci, seed=6) if w else (None, None)
    opts = dict(opts, init_trials=2)
    p_ref, _, ev_ref = oracle_mod.partition(rp, ci, k, imb, 8, vwgt=vw, ewgt=ew, options=opts, trace=True)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    p_gpu, _, ev_gpu = gp.partition(d(rp), d(ci), k, imb, 8, vwgt=d(vw), ewgt=d(ew), options=opts, trace=True)
    compare_traces(ev_ref, ev_gpu)
    p2, _, _ = gp.partition(d(rp), d(ci), k, imb, 8, vwgt=d(vw), ewgt=d(ew), options=opts)
    assert np.array_equal(p_ref, p_gpu.cpu().numpy()) and np.array_equal(p_ref, p2.cpu().numpy())


@pytest.mark.parametrize("n", [3, 8191, 8192, 8193, 16384, 16385, 2048 * 2048, 2048 * 2048 + 1])
def test_scans_of_bucket_costs(gp, cuda, n):
    """Row-cost prefixes (the scans' sizes: one block, two launches, three) through
    the exact cut and part weights of a path cut at its middle."""
    v = torch.arange(max(n - 1, 0), device=cuda)
    rp, ci = graphs.csr_from_edges(v, v + 1, n)[:2]
    k = 2
    part, st, _ = gp.partition(rp, ci, k, 0.5, 1, options={"coarsen_to": 64, "init_trials": 2})
    cut, pw = gp.edge_cut(rp, ci, part, k)
    assert cut == st["cut"] and pw.sum() == n and pw.max() == st["max_part_weight"]


@pytest.mark.parametrize("k,w", [(6, None), (300, "w")])
def test_tracked_cut_matches_oracle(oracle_mod, gp, cuda, k, w):
    """Levels of more than 4 M entries: the cut after a step comes from the moved
    rows, and rebalancing passes sweep the rows of overweight parts only; the
    iterations' cuts, proposals and partitions are the oracle's."""
    rp, ci = to_np(*graphs.grid3d(96, 100, 90))
    ew, vw = weighted(rp, ci, seed=1) if w else (None, None)
    opts = {"init_trials": 2, "coarsen_to": 100000}
    p_ref, _, ev_ref = oracle_mod.partition(rp, ci, k, 0.01, 8, vwgt=vw, ewgt=ew, options=opts, trace=True)
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    p_gpu, _, ev_gpu = gp.partition(d(rp), d(ci), k, 0.01, 8, vwgt=d(vw), ewgt=d(ew), options=opts, trace=True)
    compare_traces(ev_ref, ev_gpu)
    p2, _, _ = gp.partition(d(rp), d(ci), k, 0.01, 8, vwgt=d(vw), ewgt=d(ew), options=opts)
    assert np.array_equal(p_ref, p_gpu.cpu().numpy()) and np.array_equal(p_ref, p2.cpu().numpy())


def test_asymmetric_input_keeps_full_passes(oracle_mod, gp, cuda):
    """An input whose entries lack their mirrors (accepted, not checked by default):
    its cut is not tracked, and every iteration still equals the oracle's."""
    rp, ci = to_np(*graphs.grid3d(96, 100, 90))
    ew = np.ones(len(ci), np.int32)
    ew[::7] = 3   # weights that differ between the two directions of an edge
    opts = {"init_trials": 2, "coarsen_to": 100000, "refine_max_iters": 12}
    _, _, ev_ref = oracle_mod.partition(rp, ci, 6, 0.01, 8, ewgt=ew, options=opts, trace=True)
    d = lambda a: torch.from_numpy(a).to(cuda)
    _, _, ev_gpu = gp.partition(d(rp), d(ci), 6, 0.01, 8, ewgt=d(ew), options=opts, trace=True)
    compare_traces(ev_ref, ev_gpu)
