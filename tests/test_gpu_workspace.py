"""Device memory that a call keeps: what a small graph needs follows its own size, not
the largest grids a launch may have."""
import pytest
import torch

from thegraphpartitioning_b200 import graphs

pytestmark = pytest.mark.gpu


def test_batch_of_small_graphs_keeps_little(gp, cuda):
    specs = graphs.batch_specs(512, seed=1, nmin=1000, nmax=1001)
    gs = [graphs.batch_graph(s, device=cuda) for s in specs]
    outs = [torch.zeros(s["n"], dtype=torch.int32, device=cuda) for s in specs]
    gp.partition(gs[0][0], gs[0][1], 4, 0.03, 1)   # the library and its kernels are loaded
    gp.release_workspace()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    gp.partition_batch(gs, [s["k"] for s in specs], 0.03, [s["seed"] for s in specs], workers=1, outs=outs)
    used = free0 - torch.cuda.mem_get_info()[0]
    gp.release_workspace()
    # one worker holds all 512 hierarchies: at under 0.35 MB a graph they fit its arena's
    # first two chunks (64 and 128 MB; the scratch arena has one of 64), which 0.3 MB more
    # each would not
    assert used <= (64 + 128 + 64 + 32) << 20, used >> 20
