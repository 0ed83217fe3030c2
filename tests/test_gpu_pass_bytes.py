"""The bytes a call credits its connectivity passes with (profile = 1): whole passes
the formula of a whole sweep, rebalancing passes over the overweight parts' rows the
lists and parts of all rows, passes that end a level and sweep nothing nothing."""
import pytest
import torch

from thegraphpartitioning_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,imb,iters", [(6, 0.01, 1), (6, 0.01, 2), (6, 0.0, 3), (300, 0.0, 3)])
def test_conn_bytes_follow_what_a_pass_reads(gp, cuda, k, imb, iters):
    g = graphs.grid3d(96, 100, 90)
    rp, ci = g[0].to(cuda), g[1].to(cuda)
    opts = {"init_trials": 2, "coarsen_to": 100000, "refine_max_iters": iters}
    _, _, ev = gp.partition(rp, ci, k, imb, 8, options=opts, trace=True)
    size = {0: (rp.numel() - 1, ci.numel())}
    for e in ev:
        if e["kind"] == 2: size[e["level"] + 1] = (len(e["rowptr"]) - 1, len(e["colidx"]))
    pcb = 1 if k <= 256 else 2
    want = passes = 0
    for lv, (n, m) in size.items():
        whole = 8 * (n + 1) + 4 * m + (4 * m if lv else 0) + pcb * m + pcb * n + n + 8 * n   # coarse levels: weights
        modes = [e["mode"] for e in ev if e["kind"] == 4 and e["level"] == lv]
        tracked = m >= 1 << 22   # levels whose steps' change of the cut is known (few rows move here)
        want += whole + sum(whole if not (tracked and mode) else (4 + pcb) * n for mode in modes[1:])
        want += 0 if tracked else whole   # the pass that ends the level
        passes += len(modes) + 1
    _, s, _ = gp.partition(rp, ci, k, imb, 8, options=dict(opts, profile=1))
    assert s["conn_launches"] == passes and s["conn_bytes"] == want
