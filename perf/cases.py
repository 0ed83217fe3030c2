"""What a user of the partitioner has it do, as measurable cases.

Each case is a dict of plain values; its "op" names the public entry point:

    partition   thegraphpartitioning_b200.partition on CUDA tensors, or on host
                arrays when "host" is set (the library then copies the graph)
    batch       partition_batch over many small graphs in one call
    learned     partition_learned with the shipped scorer and its plain fallback
    score       GNN.forward: per-entry matching priorities and logits
    grad        GNN.grad of a few labelled training graphs, one call each
    cut         edge_cut of a given partition

and "family" with its sizes names the graph: R-MAT ("scale"), 2-D and 3-D grids
("x", "y", "z"), random geometric, Erdos-Renyi and Chung-Lu graphs ("n").
`listed()` gives the cases, `draw(rng)` one more of the same ranges, `prepare`
the inputs of a case from a seed, `run` one pass, `work` the bytes and
operations the pass cannot do without and `exact` the floating-point outputs
in float64 by plain torch.
"""
import math

import numpy as np
import torch

import thegraphpartitioning_b200 as gp
from thegraphpartitioning_b200 import graphs


def listed():
    return [
        # one of many small meshes or point clouds handled one by one: launches and latency
        {"name": "rgg_1500_k8", "op": "partition", "family": "rgg", "n": 1500, "k": 8, "imbalance": 0.03},
        # the small plain configuration: a 2-D five-point mesh split over four workers
        {"name": "grid512_k4", "op": "partition", "family": "grid2d", "x": 512, "y": 512, "k": 4, "imbalance": 0.03},
        # the co-purchase-shaped configuration as the command line runs it: host arrays in and out
        {"name": "copurchase_host_k64", "op": "partition", "family": "chung_lu", "n": 262111, "k": 64,
         "imbalance": 0.03, "host": True},
        # vertex and edge weights, many parts (16-bit part ids inside), a looser balance
        {"name": "rgg_weighted_k300", "op": "partition", "family": "rgg", "n": 150001, "k": 300, "imbalance": 0.05,
         "weighted": True},
        # a skewed graph of ordinary size
        {"name": "rmat20_k64", "op": "partition", "family": "rmat", "scale": 20, "k": 64, "imbalance": 0.03},
        # the headline workload, the largest
        {"name": "rmat24_k64", "op": "partition", "family": "rmat", "scale": 24, "k": 64, "imbalance": 0.03},
        # the large 3-D mesh of the evaluation set
        {"name": "grid3d_256_k32", "op": "partition", "family": "grid3d", "x": 256, "y": 256, "z": 256, "k": 32,
         "imbalance": 0.03},
        # the batched configuration's size and family mix, a thirty-second of its graphs
        {"name": "batch_128", "op": "batch", "count": 128, "nmin": 1000, "nmax": 200000, "imbalance": 0.03},
        # learned matching priorities with the plain fallback, on the evaluation family
        {"name": "learned_rmat20_k32", "op": "learned", "family": "rmat", "scale": 20, "k": 32, "imbalance": 0.03},
        # scoring every edge of a mesh once
        {"name": "score_grid3d_128", "op": "score", "family": "grid3d", "x": 128, "y": 128, "z": 128, "level": 0},
        # the gradients of a few training graphs of the training sizes
        {"name": "grad_8_graphs", "op": "grad", "count": 8, "nmin": 2000, "nmax": 64000},
        # judging a given partition of a large skewed graph
        {"name": "cut_rmat22_k64", "op": "cut", "family": "rmat", "scale": 22, "k": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, top):
    """A graph of any family with at most about top vertices (R-MAT: fewer, its rows are longer)."""
    fam = rng.choice(["rgg", "er", "chung_lu", "rmat", "grid2d", "grid3d"])
    n = _log_int(rng, 1000, top)
    if fam == "rmat":
        return {"family": fam, "scale": max(10, min(22, int(math.log2(n))))}
    if fam == "grid2d":
        x = max(16, int(math.sqrt(n) * rng.uniform(0.5, 2.0)))
        return {"family": fam, "x": x, "y": max(16, n // x)}
    if fam == "grid3d":
        x, y = (max(8, int(n ** (1 / 3) * rng.uniform(0.6, 1.6))) for _ in range(2))
        return {"family": fam, "x": x, "y": y, "z": max(4, n // (x * y))}
    return {"family": fam, "n": min(n, 1000000)}


def draw(rng):
    op = rng.choice(["partition"] * 6 + ["batch", "learned", "score", "grad", "cut"])
    if op == "batch":
        return {"op": op, "count": rng.randint(2, 160), "nmin": 1000, "nmax": _log_int(rng, 4000, 200000),
                "imbalance": 0.03}
    if op == "grad":
        return {"op": op, "count": rng.randint(1, 12), "nmin": 2000, "nmax": _log_int(rng, 4000, 64000)}
    c = {"op": op}
    c.update(_draw_graph(rng, 2000000 if op == "partition" else 1000000))
    if op == "score":
        c["level"] = rng.randint(0, 3)
        c["weighted"] = rng.random() < 0.3
        return c
    c["k"] = max(2, min(_log_int(rng, 2, 512), _size(c)[0] // 64))
    if op == "cut":
        c["weighted"] = rng.random() < 0.3
        return c
    c["imbalance"] = rng.choice([0.01, 0.03, 0.03, 0.05])
    if op == "partition":
        c["weighted"] = rng.random() < 0.25
        c["host"] = rng.random() < 0.15
    return c


# ------------------------------------------------------------------ inputs
def _size(case):
    """(vertices, directed entries) of a case's graph: exact for grids, close for the random families."""
    fam = case["family"]
    if fam == "rmat":
        s = case["scale"]
        d = 24 - s
        return int((0.529 + 0.0225 * d) * 2 ** s), int((31.04 - 0.075 * d - 0.05 * d * d) * 2 ** s)
    if fam == "grid2d":
        x, y = case["x"], case["y"]
        return x * y, 2 * (x * (y - 1) + y * (x - 1))
    if fam == "grid3d":
        x, y, z = case["x"], case["y"], case["z"]
        return x * y * z, 2 * (x * y * (z - 1) + x * z * (y - 1) + y * z * (x - 1))
    n = case["n"]
    return n, {"rgg": 8 * n, "er": 10 * n, "chung_lu": int(6.86 * n)}[fam]


def _renumbered(rowptr, colidx, shift):
    """The same mesh with its vertex numbering started `shift` vertices later (cyclic)."""
    n = rowptr.numel() - 1
    src = torch.repeat_interleave(torch.arange(n, device=rowptr.device), rowptr[1:] - rowptr[:-1])
    key = torch.sort(((src + shift) % n) * n + (colidx + shift) % n).values
    src = torch.div(key, n, rounding_mode="floor")
    rp = torch.zeros_like(rowptr)
    rp[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return rp, (key - src * n).to(torch.int32)


def _graph(case, seed):
    fam = case["family"]
    if fam == "rmat":
        return graphs.rmat(case["scale"], 16, seed=seed, device="cuda")[:2]
    if fam == "rgg":
        return graphs.random_geometric(case["n"], 8.0, seed=seed, device="cuda")
    if fam == "er":
        return graphs.erdos_renyi(case["n"], 10.0, seed=seed, device="cuda")
    if fam == "chung_lu":
        n = case["n"]
        return graphs.chung_lu(n, int(3.43 * n), 2.5, max(20.0, 420.0 * n / 262111), seed=seed, device="cuda")
    rp, ci = (graphs.grid2d(case["x"], case["y"], device="cuda") if fam == "grid2d" else
              graphs.grid3d(case["x"], case["y"], case["z"], device="cuda"))
    return _renumbered(rp, ci, (seed * 7919 + 13) % (rp.numel() - 1))


def _weights(rp, ci, seed):
    """Vertex weights 1..8 and symmetric edge weights 1..16."""
    n = rp.numel() - 1
    g = torch.Generator(device="cuda").manual_seed(seed)
    vw = torch.randint(1, 9, (n,), generator=g, device="cuda", dtype=torch.int32)
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
    a, b = torch.minimum(src, ci.long()), torch.maximum(src, ci.long())
    ew = (1 + (a * 40503 + b * 9973 + (a * b >> 3) + seed) % 16).to(torch.int32)
    return vw, ew


def _scorer_params(seed):
    """He-scaled weights of the edge scorer (float32), every block and edge coefficient non-zero."""
    rng = np.random.default_rng(seed + 77)
    blocks = [(64 * 8, 0.5), (64, 0.05), (8 * 64, 0.125), (64 * 72, 0.1667), (64, 0.05), (4 * 64, 0.125), (4, 0.1)]
    p = np.concatenate([rng.normal(0, s, c) for c, s in blocks] + [[1.0, 0.3, 0.1, 0.28]])
    return p.astype(np.float32)


def _training_graph(i, nmin, nmax, seed):
    """One labelled level of a training graph: (rowptr, colidx, vwgt, ewgt, level, label); an entry is
    labelled 1 when both ends fall into the same of 16 id blocks or (one in four) by a hash."""
    rng = np.random.default_rng(i)   # sizes belong to the case, contents to the seed
    n = int(round(math.exp(rng.uniform(math.log(nmin), math.log(nmax)))))
    fam = ("chung_lu", "rmat", "rgg", "er")[i % 4]
    case = {"family": fam, "scale": max(10, int(round(math.log2(n)))) if fam == "rmat" else 0, "n": n}
    rp, ci = _graph(case, seed * 131 + i)
    vw, ew = _weights(rp, ci, seed + i) if i % 2 else (None, None)   # coarse levels carry weights
    n = rp.numel() - 1
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
    dst = ci.long()
    same = (src * 16 // n) == (dst * 16 // n)
    label = torch.where((src + dst) * 2654435761 % 4 == 0, (src + dst) % 3 == 0, same).to(torch.uint8)
    return rp, ci, vw, ew, (i // 4) % 4 if vw is not None else 0, label


def _host(t):
    return None if t is None else t.cpu().numpy()


def _most(case):
    """(vertices, directed entries) that no seed of a case's random graph exceeds; a program that handles
    such graphs one after another keeps its result buffers that large."""
    n, m = _size(case)
    if case["family"] in ("grid2d", "grid3d"):
        return n, m
    n = 2 ** case["scale"] if case["family"] == "rmat" else case["n"]
    return n, 32 * n if case["family"] == "rmat" else 12 * n


def prepare(case, seed):
    op = case["op"]
    st = {"case": case, "op": op, "seed": seed}
    if op == "batch":
        # sizes and parts of the configuration's mix belong to the case, contents to the seed
        specs = graphs.batch_specs(case["count"], seed=0, nmin=case["nmin"], nmax=case["nmax"])
        st["seeds"] = [s["seed"] + seed for s in specs]
        st["graphs"] = [graphs.batch_graph(dict(s, seed=x), device="cuda") for s, x in zip(specs, st["seeds"])]
        st["ks"] = [s["k"] for s in specs]
        st["parts"] = torch.zeros(sum(s["n"] for s in specs), dtype=torch.int32, device="cuda")
        st["outs"] = list(torch.split(st["parts"], [s["n"] for s in specs]))
    elif op == "grad":
        st["samples"] = [_training_graph(i, case["nmin"], case["nmax"], seed) for i in range(case["count"])]
        st["model"] = gp.GNN(_scorer_params(seed))
    else:
        st["rp"], st["ci"] = _graph(case, seed)
        st["vw"], st["ew"] = _weights(st["rp"], st["ci"], seed) if case.get("weighted") else (None, None)
        n = st["rp"].numel() - 1
        if op == "cut":
            g = torch.Generator(device="cuda").manual_seed(seed)
            st["part"] = torch.randint(0, case["k"], (n,), generator=g, device="cuda", dtype=torch.int32)
        elif op == "score":
            st["model"] = gp.GNN(_scorer_params(seed))
            st["prio"] = torch.zeros(_most(case)[1], dtype=torch.int32, device="cuda")
            st["logit"] = torch.zeros(_most(case)[1], device="cuda")
        elif case.get("host"):
            for key in ("rp", "ci", "vw", "ew"):
                st[key] = _host(st[key])
            st["part"] = np.zeros(_most(case)[0], dtype=np.int32)
        else:
            if op == "learned":
                st["model"] = gp.default_gnn()
            st["part"] = torch.zeros(_most(case)[0], dtype=torch.int32, device="cuda")
            st["out"] = st["part"][:n]
    # the generators' scratch goes back to the device: the library allocates outside torch's pool
    torch.cuda.empty_cache()
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    case, op = st["case"], st["op"]
    if op == "partition":
        part, stats, _ = gp.partition(st["rp"], st["ci"], case["k"], imbalance=case["imbalance"], seed=st["seed"],
                                      vwgt=st["vw"], ewgt=st["ew"], out=st.get("out"))
        if case.get("host"):
            st["part"][:part.shape[0]] = part
        return {"part": st["part"], "cut": stats["cut"], "max_part_weight": stats["max_part_weight"]}
    if op == "batch":
        _, stats = gp.partition_batch(st["graphs"], st["ks"], case["imbalance"], st["seeds"], outs=st["outs"])
        return {"parts": st["parts"], "cuts": np.array([s["cut"] for s in stats])}
    if op == "learned":
        _, stats, report, _ = gp.partition_learned(st["rp"], st["ci"], case["k"], st["model"],
                                                   imbalance=case["imbalance"], seed=st["seed"], out=st["out"])
        return {"part": st["part"], "cut": stats["cut"], "cut_learned": report["cut_learned"],
                "cut_plain": report["cut_plain"]}
    if op == "score":
        prio, logit = st["model"].forward(st["rp"], st["ci"], st["vw"], st["ew"], level=case["level"])
        if case["family"] in ("grid2d", "grid3d"):
            return {"prio": prio, "logit": logit}
        st["prio"][:prio.numel()] = prio      # the number of entries depends on the seed
        st["logit"][:logit.numel()] = logit
        return {"prio": st["prio"], "logit": st["logit"]}
    if op == "grad":
        res = [st["model"].grad(rp, ci, label, vw, ew, level=level)
               for rp, ci, vw, ew, level, label in st["samples"]]
        return {"loss": np.array([r[0] for r in res]), "grad": np.stack([r[1] for r in res])}
    cut, pw = gp.edge_cut(st["rp"], st["ci"], st["part"], case["k"], ewgt=st["ew"], vwgt=st["vw"])
    return {"cut": cut, "part_weights": pw}


def _graph_bytes(n, m, weighted):
    return 8 * (n + 1) + 4 * m + (4 * n + 4 * m if weighted else 0)


def work(case):
    op = case["op"]
    if op in ("batch", "grad"):
        lo, hi = case["nmin"], case["nmax"]
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo   # of a log-uniform size
        n = int(case["count"] * mean)
        m = 9 * n if op == "batch" else 13 * n
        if op == "batch":
            return {"bytes": _graph_bytes(n, m, False) + 4 * n, "flops": 0}
        return {"bytes": _graph_bytes(n, m, False) + (4 * n + 4 * m) // 2 + m, "flops": 3 * _score_flops(n, m)}
    n, m = _size(case)
    g = _graph_bytes(n, m, case.get("weighted"))
    if op == "score":
        return {"bytes": g + 8 * m, "flops": _score_flops(n, m)}
    return {"bytes": g + 4 * n, "flops": 0}


def _score_flops(n, m):
    """Two layers (64 x 8 and 64 x 72), their projections (8 x 64 and 4 x 64) per vertex; the means of 4
    and 8 floats and the logit per entry."""
    return n * 2 * (64 * 8 + 8 * 64 + 64 * 72 + 4 * 64) + m * 32


# ------------------------------------------------------------------ float64 values
def _bit(ids):
    """Signature bit 0..127 of each vertex id (int64): the top 7 bits of fmix32(id * 0x9E3779B1)."""
    mask = 0xFFFFFFFF
    x = (ids * 0x9E3779B1) & mask
    x = x ^ (x >> 16)
    x = (x * 0x85EBCA6B) & mask
    x = x ^ (x >> 13)
    x = (x * 0xC2B2AE35) & mask
    x = x ^ (x >> 16)
    return x >> 25


def _common(src, col, n):
    """Common-neighbour counts through 128-bit signatures, without the two ends' own bits."""
    sig = torch.zeros(n, 128, dtype=torch.bool, device=src.device)
    sig[src, _bit(col)] = True
    out = torch.empty(src.numel(), dtype=torch.float64, device=src.device)
    for a in range(0, src.numel(), 1 << 22):
        s, d = src[a:a + (1 << 22)], col[a:a + (1 << 22)]
        both = sig[s] & sig[d]
        at = torch.arange(s.numel(), device=src.device)
        both[at, _bit(s)] = False
        both[at, _bit(d)] = False
        out[a:a + (1 << 22)] = both.sum(1)
    return out


def _logits(p, rp, ci, vw, ew, level):
    """Edge logits of the scorer with parameters p (a float64 tensor already rounded to bfloat16)."""
    H, F, M, Z = 64, 4, 8, 4
    w1, b1, pm, w2, b2, z, a, edge = torch.split(p, [H * 2 * F, H, M * H, H * (H + M), H, Z * H, Z, 4])
    n = rp.numel() - 1
    deg_i = rp[1:] - rp[:-1]
    src, col = torch.repeat_interleave(torch.arange(n, device=rp.device), deg_i), ci.long()
    one = lambda c: torch.ones(c, dtype=torch.float64, device=rp.device)
    w = one(col.numel()) if ew is None else ew.double()
    v = one(n) if vw is None else vw.double()
    deg = deg_i.double()
    inv = torch.where(deg > 0, 1 / deg.clamp(min=1), torch.zeros_like(deg))[:, None]
    mean = lambda x: torch.zeros(n, x.shape[1], dtype=torch.float64, device=rp.device).index_add(0, src, x[col]) * inv
    wdeg = torch.zeros(n, dtype=torch.float64, device=rp.device).index_add(0, src, w)
    x = torch.stack([torch.log2(1 + deg) / 8, torch.log2(1 + wdeg) / 16, torch.log2(1 + v) / 16,
                     one(n) * (level / 16)], 1)
    h1 = torch.relu(torch.cat([x, mean(x)], 1) @ w1.view(H, 2 * F).T + b1)
    h2 = torch.relu(torch.cat([h1, mean(h1 @ pm.view(M, H).T)], 1) @ w2.view(H, H + M).T + b2)
    zz = h2 @ z.view(Z, H).T
    return ((zz[src] * zz[col] * a).sum(1) + edge[0] * torch.log2(1 + w) / 8
            + edge[1] * (w / wdeg[src] + w / wdeg[col]) + edge[2]
            + edge[3] * torch.log2(1 + _common(src, col, n)) / 7)


def exact(case, seed):
    op = case["op"]
    if op not in ("score", "grad"):
        return None   # whole numbers
    p = torch.from_numpy(_scorer_params(seed)).cuda().bfloat16().double()
    if op == "score":
        rp, ci = _graph(case, seed)
        vw, ew = _weights(rp, ci, seed) if case.get("weighted") else (None, None)
        with torch.no_grad():
            t = _logits(p, rp, ci, vw, ew, case["level"])
        return {"prio": None, "logit": torch.nn.functional.pad(t, (0, _most(case)[1] - t.numel()))}
    losses, grads = [], []
    for i in range(case["count"]):
        rp, ci, vw, ew, level, label = _training_graph(i, case["nmin"], case["nmax"], seed)
        q = p.clone().requires_grad_(True)
        loss = torch.nn.functional.binary_cross_entropy_with_logits(_logits(q, rp, ci, vw, ew, level), label.double())
        loss.backward()
        losses.append(float(loss))
        grads.append(q.grad.cpu().numpy())
    return {"loss": np.array(losses), "grad": np.stack(grads)}
