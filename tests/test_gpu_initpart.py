"""Initial partition against the oracle where its dispatch can go wrong.

No coarsening (coarsen_to = n), so the initial partition sees the graph as it
is; the kept trial and its labels are compared exactly with the oracle's.
"""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from thegraphpartitioning_b200._abi import GP_TR_INITPART
from helpers import to_np, weighted

pytestmark = pytest.mark.gpu


def _dense(n, deg, seed):
    """deg hashed neighbours per vertex: mean degree about 2 * deg (large frontiers)."""
    return graphs.erdos_renyi(n, 2.0 * deg, seed=seed)


def _pieces(n, piece):
    """Disjoint paths of `piece` vertices: most of a label is unreached by its BFS."""
    src = torch.arange(n - 1)
    src = src[(src + 1) % piece != 0]
    return graphs.csr_from_edges(src, src + 1, n)[:2]


def _cases():
    yield "n2_k2", graphs.path(2), 2, None, 64
    yield "n17_k16", graphs.path(17), 16, None, 64
    yield "k_is_n_w", graphs.path(9), 9, "w", 8                     # labels without vertices
    yield "path4095_k3", graphs.path(4095), 3, None, 4             # 4095 BFS levels
    yield "pieces_k7", _pieces(1000, 3), 7, "w", 64
    yield "rows_on_chip_w", graphs.random_geometric(1500, 8.0, seed=1), 33, "w", 64
    yield "tile16_k300", graphs.erdos_renyi(8864, 14.0, seed=2), 300, "w", 8
    yield "dense_bottom_up", _dense(2000, 100, 3), 64, None, 8
    yield "dense_w_k2", _dense(700, 150, 4), 2, "w", 33
    yield "lists_off_chip", graphs.grid2d(160, 205), 5, None, 4    # 32,800 vertices: state on chip, lists not
    yield "k1024", graphs.erdos_renyi(9000, 6.0, seed=5), 1024, None, 4
    yield "ids_16bit_last", graphs.erdos_renyi(50000, 6.0, seed=6), 6, None, 2
    yield "general_kernel", graphs.erdos_renyi(65535, 6.0, seed=7), 6, None, 2


CASES = list(_cases())


@pytest.mark.parametrize("name,g,k,w,trials", CASES, ids=[c[0] for c in CASES])
def test_initial_partition_matches_oracle(oracle_mod, gp, cuda, name, g, k, w, trials):
    rp, ci = to_np(*g)
    ew, vw = weighted(rp, ci, seed=3) if w else (None, None)
    opts = {"coarsen_to": max(len(rp), 2), "init_trials": trials, "refine_max_iters": 1}
    _, s_ref, ev = oracle_mod.partition(rp, ci, k, 0.1, 5, vwgt=vw, ewgt=ew, options=opts, trace=True)
    ref = [e for e in ev if e["kind"] == GP_TR_INITPART][0]
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    _, s_gpu, ev = gp.partition(d(rp), d(ci), k, 0.1, 5, vwgt=d(vw), ewgt=d(ew), options=opts,
                                trace={GP_TR_INITPART})
    assert s_gpu["levels"] == 1 and s_gpu["best_trial"] == s_ref["best_trial"]
    for key in ("iter", "cut", "maxpw"):
        assert ev[0][key] == ref[key], key
    assert np.array_equal(ev[0]["a0"], ref["a0"])
