"""Contraction of long rows at the edges of its one-block tiers (512, 2048, 4096,
12288, 65536 walk entries) and at the coarse sizes where their table slots go from
32 to 64 bits (2^16, 2^18, 2^20, 2^21 vertices): every hub's coarse row against
the definition (mapped ids of both members' rows in order of first occurrence,
summed weights, itself left out)."""
import numpy as np
import pytest
import torch

from thegraphpartitioning_b200 import graphs
from thegraphpartitioning_b200._abi import GP_TR_CONTRACT
from helpers import to_np, weighted

pytestmark = pytest.mark.gpu


def _hubs(n, degs):
    """A ring with hubs: hub i (vertex 50 i) linked to degs[i] vertices spread over the ring."""
    v = torch.arange(n)
    a, b = [v], [(v + 1) % n]
    for i, d in enumerate(degs):
        g = torch.Generator().manual_seed(1000 + i)
        t = torch.randperm(n, generator=g)[:d]
        a.append(torch.full((d,), 50 * i))
        b.append(t[t != 50 * i])
        a[-1] = a[-1][:len(b[-1])]
    return graphs.csr_from_edges(torch.cat(a), torch.cat(b), n)[:2]


EDGES = [505, 511, 515, 2040, 2046, 2052, 4088, 4094, 4100, 12280, 12286, 12292, 30000]
CASES = [("n90k_w", 90_000, EDGES + [65528, 65534, 65540], True),       # coarse size below 2^16
         ("n140k", 140_000, EDGES + [50000, 65534, 65540, 100000], False),   # above it
         ("n480k_w", 480_000, EDGES, True), ("n600k", 600_000, EDGES, False),          # 2^18
         ("n1900k", 1_900_000, EDGES, False), ("n2300k_w", 2_300_000, EDGES, True),    # 2^20
         ("n4700k", 4_700_000, EDGES, False)]                                          # 2^21


@pytest.mark.parametrize("name,n,degs,w", CASES, ids=[c[0] for c in CASES])
def test_hub_rows_contract_exactly(gp, cuda, name, n, degs, w):
    rp, ci = to_np(*_hubs(n, degs))
    ew = weighted(rp, ci, seed=5)[0] if w else np.ones(len(ci), np.int32)
    d = lambda a: torch.from_numpy(a).to(cuda)
    opts = dict(coarsen_to=int(0.7 * n), init_trials=1, refine_max_iters=1)
    _, _, ev = gp.partition(d(rp), d(ci), 2, 0.5, 4, ewgt=d(ew) if w else None, options=opts, trace={GP_TR_CONTRACT})
    e = [x for x in ev if x["kind"] == GP_TR_CONTRACT][0]
    cmap, crp, cci, cew = e["a0"], e["rowptr"], e["colidx"], e["ewgt"]
    order = np.argsort(cmap, kind="stable")          # members of each coarse vertex, lower id first
    first = np.searchsorted(cmap[order], np.arange(len(crp)))
    for c in np.unique(cmap[50 * np.arange(len(degs))]):
        mem = order[first[c]:first[c + 1]]
        assert 1 <= len(mem) <= 2
        ids = np.concatenate([cmap[ci[rp[v]:rp[v + 1]]] for v in mem])
        ws = np.concatenate([ew[rp[v]:rp[v + 1]] for v in mem]).astype(np.int64)
        keep = ids != c
        u, at, inv = np.unique(ids[keep], return_index=True, return_inverse=True)
        sums = np.bincount(inv, weights=ws[keep], minlength=len(u))
        o = np.argsort(at, kind="stable")
        assert np.array_equal(cci[crp[c]:crp[c + 1]], u[o])
        assert np.array_equal(cew[crp[c]:crp[c + 1]], sums[o].astype(np.int64))
