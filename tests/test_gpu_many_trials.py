"""More trials of the initial partition than 16 times the rows of a grid (1,048,560):
the trials then add up their own cuts; the kept one is no worse than the best of few."""
import pytest
import torch

from thegraphpartitioning_b200 import graphs

pytestmark = pytest.mark.gpu


def test_a_million_trials(gp, cuda):
    rp, ci = (x.to(cuda) for x in graphs.erdos_renyi(700, 130.0, seed=3)[:2])
    assert ci.numel() >= 65536   # where the trials' cuts are otherwise summed together
    one = gp.partition(rp, ci, 2, 0.03, 1, options={"init_trials": 64, "refine_max_iters": 1})[1]
    part, many, _ = gp.partition(rp, ci, 2, 0.03, 1, options={"init_trials": 65535 * 16 + 1, "refine_max_iters": 1})
    assert gp.edge_cut(rp, ci, part, 2)[0] == many["cut"] and many["max_part_weight"] <= many["max_allowed"]
    gp.release_workspace()
    assert many["best_trial"] >= 0 and many["cut"] <= 1.02 * one["cut"]
