"""The bounds-checked build over what its other test is too small to reach: the
cut's change from the moved rows and the passes after it (levels of 4 M entries),
candidates collected 32 vertices per thread (1 M vertices), contraction tables of
64-bit slots (coarse ids of 16 to 21 bits and more beside long rows).  No index out
of range, and the oracle's partitions."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import sys
import numpy as np
import torch
sys.path.insert(0, ROOT); sys.path.insert(0, ROOT + "/tests")
import oracle
import thegraphpartitioning_b200 as gp
from thegraphpartitioning_b200 import graphs
from helpers import multi_star_grid, to_np
assert gp.CHECKED and gp.LIB_PATH.endswith("libgp_b200_checked.so")
dev = torch.device("cuda:0")
gp.checked_violations(clear=True)
rm, g3 = to_np(*graphs.rmat(18, seed=6)[:2]), to_np(*graphs.grid3d(96, 100, 90))
assert len(rm[1]) > 1 << 22 and len(g3[1]) > 1 << 22
g2 = to_np(*graphs.grid2d(1024, 1031))
cases = [
    (rm, 64, 0.01, {"refine_max_iters": 9}), (rm, 300, 0.05, {"refine_max_iters": 4}),
    (g3, 6, 0.01, {}), (g3, 300, 0.0, {"refine_max_iters": 6}),
    (g2, 2, 0.0, {"refine_max_iters": 3}), (g2, 260, 0.0, {"refine_max_iters": 3}),
    (to_np(*multi_star_grid(side=2100)), 2, 0.03, {"refine_max_iters": 1}),
]
for (rp, ci), k, imb, opts in cases:
    opts = dict(opts, init_trials=2)
    ref, rst, _ = oracle.partition(rp, ci, k, imb, 5, options=opts)
    got, st, _ = gp.partition(torch.from_numpy(rp).to(dev), torch.from_numpy(ci).to(dev), k, imb, 5, options=opts)
    assert np.array_equal(ref, got.cpu().numpy()) and st["cut"] == rst["cut"], (len(rp), k)
cnt, site = gp.checked_violations(clear=True)
print("violations", cnt, "first site", site)
assert cnt == 0, (cnt, site)
'''


def test_bounds_checked_build_on_large_levels(gp, cuda, oracle_mod):
    env = dict(os.environ, THEGRAPHPARTITIONING_CHECKED="1")
    out = subprocess.run([sys.executable, "-c", CHILD.replace("ROOT", repr(ROOT))], env=env, capture_output=True,
                         text=True, timeout=900)
    assert out.returncode == 0, out.stdout[-3000:] + out.stderr[-3000:]
    assert "violations 0" in out.stdout


@pytest.fixture(scope="module")
def star_grid():
    from helpers import multi_star_grid, to_np
    return to_np(*multi_star_grid(side=2100))


def test_long_rows_beside_many_coarse_vertices(gp, cuda, oracle_mod, star_grid):
    """The coarse graph of a contraction whose tables need 64-bit slots in every tier."""
    import numpy as np
    import torch
    from helpers import compare_traces
    rp, ci = star_grid
    opts = {"init_trials": 2, "refine_max_iters": 1, "match_rounds": 2}
    _, _, ev_ref = oracle_mod.partition(rp, ci, 2, 0.03, 8, options=opts, trace=True)
    first = next(e for e in ev_ref if e["kind"] == 2)
    assert len(first["rowptr"]) - 1 >= 1 << 21 and np.diff(first["rowptr"]).max() > 65536
    _, _, ev_gpu = gp.partition(torch.from_numpy(rp).to(cuda), torch.from_numpy(ci).to(cuda), 2, 0.03, 8, options=opts,
                                trace=True)
    compare_traces(ev_ref, ev_gpu)
