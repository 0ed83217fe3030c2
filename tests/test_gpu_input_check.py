"""What the input check reports: the message with the exact entry or row, for an id
out of range, a self-loop and a weight below 1, at the edges of lanes, of windows of
32 rows and of slices, on rows short and long enough for both widths of the pass."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(name, n):
    rng = np.random.default_rng(n)
    if name == "ragged":
        deg = rng.integers(0, 40, n)
        deg[rng.integers(0, n, n // 5)] = 0      # empty rows between
        deg[0], deg[n // 2], deg[-1] = 3, 5000, 2   # and one longer than slices
    else:
        deg = np.full(n, int(name))
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    src = np.repeat(np.arange(n), deg)
    ci = ((src + 1 + rng.integers(0, n - 1, len(src))) % n).astype(np.int32)   # never the row itself
    return rp, ci, src


@pytest.mark.parametrize("name,n", [("4", 33), ("4", 4099), ("12", 3001), ("40", 2003), ("ragged", 2500)])
def test_bad_entries_are_named(gp, cuda, name, n):
    rp, ci, src = _graph(name, n)
    m = len(ci)
    d = lambda a: torch.from_numpy(a).to(cuda)

    def message(ci, ew=None):
        with pytest.raises(gp.GPError) as e:
            gp.partition(d(rp), d(ci), 2, 0.1, 1, ewgt=None if ew is None else d(ew))
        return str(e.value)

    at = sorted({e for e in (0, 1, 31, 32, 127, 128, 129, 191, 192, 255, 256, 257, 511, 512, m // 2, int(rp[n // 2]),
                             int(rp[n // 2 + 1]) - 1, m - 33, m - 2, m - 1) if 0 <= e < m})
    for e in at:
        for bad in (n, -1, 2 ** 31 - 1):
            x = ci.copy(); x[e] = bad
            assert message(x).endswith(f"column index out of range at entry {e}"), (e, bad)
        x = ci.copy(); x[e] = src[e]
        assert message(x).endswith(f"self-loop at vertex {src[e]}"), e
        for bad in (0, -5):
            w = np.ones(m, np.int32); w[e] = bad
            assert message(ci, w).endswith(f"edge weight < 1 at entry {e}"), (e, bad)
    # of several, the smallest code (ids, then self-loops, then weights), then the first
    a, b, c = at[2], at[len(at) // 2], at[-1]
    x = ci.copy(); x[c] = n; x[b] = n; x[a] = src[a]
    w = np.ones(m, np.int32); w[0] = 0
    assert message(x, w).endswith(f"column index out of range at entry {b}")
