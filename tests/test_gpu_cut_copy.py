"""The exact cut around the size from which it gathers from a byte copy of the parts
(4,194,304 entries, up to 256 parts, a mean degree of 8): cut and part weights against
numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [False, True])
@pytest.mark.parametrize("n,deg,k", [(524287, 8, 256), (524288, 8, 256), (524288, 8, 257), (599187, 7, 64), (70001, 61, 5)])
def test_cut_from_bytes_matches_numpy(gp, cuda, n, deg, k, w):
    rng = np.random.default_rng(n + k)
    m = n * deg
    rp = np.arange(n + 1, dtype=np.int64) * deg
    ci = rng.integers(0, n, m).astype(np.int32)
    part = rng.integers(0, k, n).astype(np.int32)
    part[:2] = k - 1, 0
    ew = rng.integers(1, 100, m).astype(np.int32) if w else None
    vw = rng.integers(1, 100, n).astype(np.int32) if w else None
    apart = np.repeat(part, deg) != part[ci]
    cross = int(ew[apart].sum(dtype=np.int64) if w else apart.sum())
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    cut, pw = gp.edge_cut(d(rp), d(ci), d(part), k, ewgt=d(ew), vwgt=d(vw))
    assert cut == cross // 2
    assert np.array_equal(np.asarray(pw), np.bincount(part, weights=vw, minlength=k).astype(np.int64))
