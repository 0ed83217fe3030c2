"""Batches of graphs around the entry count up to which one block refines a level:
the partitions are those of single calls."""
import pytest
import torch

from thegraphpartitioning_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degs", [(4000, (15.0, 16.0, 16.3, 16.5, 17.0, 60.0)), (16000, (3.5, 4.0, 4.1, 4.2, 8.0)),
                                    (60000, (1.0, 1.1, 6.0))])
def test_batch_around_the_entry_limit(gp, cuda, n, degs):
    gs = [tuple(t.to(cuda) for t in graphs.erdos_renyi(n, d, seed=i)[:2]) for i, d in enumerate(degs)]
    if n < 20000:
        ms = [g[1].numel() for g in gs]
        assert min(ms) <= 65536 < max(ms)
    ks, seeds = [4 + i for i in range(len(gs))], list(range(len(gs)))
    parts, stats = gp.partition_batch(gs, ks, 0.03, seeds, workers=3)
    for (rp, ci), k, seed, part, st in zip(gs, ks, seeds, parts, stats):
        one, s, _ = gp.partition(rp, ci, k, 0.03, seed)
        assert torch.equal(one, part) and s["cut"] == st["cut"]
