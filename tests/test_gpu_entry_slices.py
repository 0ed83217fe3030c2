"""Entry-sliced passes where a window of 32 rows holds fewer, exactly or more than
256 entries, runs of empty rows, rows longer than a slice, and both widths the cut
gathers from: cut and part weights against numpy, validation at the last entry."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _degrees(name, n, rng):
    if name == "six": return np.full(n, 6)
    if name == "eight": return np.full(n, 8)              # windows of exactly 256
    if name == "nine": return np.full(n, 9)
    if name == "ragged": return rng.integers(0, 40, n)
    if name == "empty_runs":
        d = rng.integers(0, 12, n)
        d[np.arange(n) // 97 % 3 != 0] = 0
        d[0] = d[-1] = 0
        return d
    d = rng.integers(0, 5, n)                             # "hubs": rows longer than a slice
    d[[3, n // 2, n - 1]] = [70000, 16384, 33000]
    return d


CASES = [("six", 1, 2), ("six", 20011, 7), ("eight", 32768, 5), ("eight", 140_000, 256), ("nine", 140_001, 257),
         ("ragged", 60_000, 64), ("ragged", 33, 3), ("empty_runs", 100_003, 9), ("hubs", 50_000, 16), ("ragged", 400_000, 300)]


@pytest.mark.parametrize("w", [False, True])
@pytest.mark.parametrize("name,n,k", CASES)
def test_cut_matches_numpy(gp, cuda, name, n, k, w):
    rng = np.random.default_rng(n + k)
    deg = _degrees(name, n, rng)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    m = int(rp[-1])
    ci = rng.integers(0, n, m).astype(np.int32)
    part = rng.integers(0, k, n).astype(np.int32)
    ew = rng.integers(1, 100, m).astype(np.int32) if w else None
    vw = rng.integers(1, 100, n).astype(np.int32) if w else None
    src = np.repeat(np.arange(n), deg)
    cross = int((part[src] != part[ci]).astype(np.int64) @ (ew if w else np.ones(m, np.int64)).astype(np.int64))
    d = lambda a: None if a is None else torch.from_numpy(a).to(cuda)
    cut, pw = gp.edge_cut(d(rp), d(ci), d(part), k, ewgt=d(ew), vwgt=d(vw))
    assert cut == cross // 2
    assert np.array_equal(np.asarray(pw), np.bincount(part, weights=vw, minlength=k).astype(np.int64))


@pytest.mark.parametrize("n", [33, 4099])
def test_bad_entry_is_reported_wherever_it_is(gp, cuda, n):
    v = torch.arange(n)
    from thegraphpartitioning_b200 import graphs
    rp, ci = graphs.csr_from_edges(torch.cat([v, v]), torch.cat([(v + 1) % n, (v + 5) % n]), n)[:2]
    for e in (0, 31, 32, len(ci) // 2, len(ci) - 1):
        bad = ci.clone()
        bad[e] = n
        with pytest.raises(Exception):
            gp.partition(rp.to(cuda), bad.to(cuda), 2, 0.1, 1)
    gp.partition(rp.to(cuda), ci.to(cuda), 2, 0.1, 1)
