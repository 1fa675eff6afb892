"""The work a user of this library has it do, as cases that can be timed one by one.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges.  ``prepare`` makes a
case's inputs on the GPU (or, for the drop-in call, on the host) together with the workspace or
plan a program keeps between calls; ``run`` is one pass through the public entry points; ``work``
counts the bytes and operations the pass cannot do without; ``exact`` is the same result in 64 bits
from plain torch.

The embeddings are Gaussian mixtures like those of ``msc_b200.synth`` (cluster centres N(0, 25) per
dimension, unit spread within, optionally LogNormal cluster sizes, anisotropic spreads, 1% uniform
noise cells, rows L2-normalised for the cosine metric), drawn on the GPU.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "metal-singlecell_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from msc_b200 import batch as mbatch                      # noqa: E402
from msc_b200 import bbknn as mbb                         # noqa: E402
from msc_b200 import neighbors as nbm                     # noqa: E402
from msc_b200 import spatial as msp                       # noqa: E402

DEV = "cuda"


def listed():
    return [
        # the smallest request a graph service sees: a few hundred cells (the size of the
        # reference's own parity input); launches and host work are all of it
        _graph("graph_500", 500, 20, 15, clusters=5),
        # an ordinary single sample, scanpy's defaults
        _graph("graph_10k", 10_000, 50, 15, clusters=20),
        # an odd size with wide rows (100 PCs), the cosine metric and the Gaussian kernel
        _graph("graph_31k_wide_gauss", 31_007, 100, 10, clusters=25, metric="cosine",
               method="gauss"),
        # a large study: cosine, 30 neighbours, clusters of different shapes and sizes
        _graph("graph_200k_cosine", 200_000, 50, 30, clusters=50, sizes=1.0, aniso=True,
               metric="cosine"),
        # an atlas: 1.3 million cells with 1% of noise cells
        _graph("graph_1m3", 1_300_000, 50, 15, clusters=200, sizes=1.0, noise=0.01),
        # the call with the embedding on the host: pinned memory in, both matrices in pinned memory
        # out, copies overlapped
        _graph("host_100k", 100_000, 50, 15, clusters=60, sizes=1.0, noise=0.01, kind="host"),
        # the neighbour search of doublet detection: 3,000 observed and 6,000 simulated cells,
        # many neighbours
        _graph("knn_9k_wide_list", 9_000, 30, 82, clusters=10, kind="knn", doublets=True),
        # a cohort: 64 samples of 2,000 to 100,000 cells (30 PCs) searched in one launch
        {"name": "cohort_64", "kind": "cohort", "samples": 64, "median": 11_000, "d": 30, "k": 15,
         "shape_seed": 3},
        # a batch-balanced graph over eight batches
        {"name": "bbknn_200k", "kind": "bbknn", "n": 200_000, "d": 50, "batches": 8, "within": 3,
         "clusters": 50},
        # a spatial slide of a million spots: nearest neighbours, and all within a radius
        {"name": "spatial_knn_1m", "kind": "spatial_knn", "n": 1_000_000, "k": 7},
        {"name": "spatial_radius_250k", "kind": "spatial_radius", "n": 250_003, "radius": 30.0},
        # the hand-off to the UMAP layout: weak edges pruned, sampling periods
        {"name": "umap_edges_200k", "kind": "umap_edges", "n": 200_000, "k": 15},
    ]


def draw(rng):
    kind = rng.choice(["graph"] * 6 + ["host", "knn", "knn", "cohort", "bbknn", "spatial_knn",
                                       "spatial_radius", "umap_edges"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind in ("graph", "host"):
        n = size(500, 400_000) if kind == "graph" else size(2_000, 200_000)
        metric = rng.choice(["euclidean", "euclidean", "cosine"])
        return _graph(None, n, rng.choice([10, 20, 30, 50, 50, 100, rng.randint(5, 100)]),
                      rng.choice([10, 15, 15, 30, rng.randint(5, 33)]),
                      clusters=max(1, min(200, int(n ** 0.4 * rng.uniform(0.5, 1.5)))),
                      sizes=rng.choice([0.0, 0.5, 1.0]), noise=rng.choice([0.0, 0.0, 0.01]),
                      aniso=rng.random() < 0.3, metric=metric,
                      method=rng.choice(["umap", "umap", "umap", "gauss"]), kind=kind,
                      precision=rng.choice(["fp16", "fp16", "fp16", "bf16x3"]))
    if kind == "knn":
        if rng.random() < 0.5:          # doublet detection: k = round(1.5·√n) + 1 of 3n cells
            n = size(1_000, 8_000)
            return _graph(None, 3 * n, 30, int(round(1.5 * math.sqrt(n))) + 1, clusters=10,
                          kind="knn", doublets=True)
        return _graph(None, size(500, 300_000), rng.randint(5, 100), rng.randint(5, 65),
                      clusters=rng.randint(5, 60), sizes=0.5, kind="knn")
    if kind == "cohort":
        return {"kind": "cohort", "samples": rng.randint(4, 64), "median": size(3_000, 11_000),
                "d": rng.choice([30, 50]), "k": rng.choice([10, 15, 30]),
                "shape_seed": rng.randint(0, 10_000)}
    if kind == "bbknn":
        return {"kind": "bbknn", "n": size(3_000, 200_000), "d": rng.choice([30, 50]),
                "batches": rng.randint(2, 12), "within": rng.randint(2, 6),
                "clusters": rng.randint(5, 50)}
    if kind == "spatial_knn":
        return {"kind": "spatial_knn", "n": size(3_000, 1_000_000), "k": rng.randint(4, 31)}
    if kind == "spatial_radius":
        n = size(3_000, 400_000)
        # a radius with about 4 to 40 points of the uniform background in it
        return {"kind": "spatial_radius", "n": n,
                "radius": round(10_000 * math.sqrt(size(4, 40) / (math.pi * n)), 2)}
    return {"kind": "umap_edges", "n": size(2_000, 800_000), "k": rng.randint(10, 30)}


def _graph(name, n, d, k, *, clusters, sizes=0.0, noise=0.0, aniso=False, metric="euclidean",
           method="umap", kind="graph", precision="fp16", doublets=False):
    c = dict(kind=kind, n=n, d=d, k=k, clusters=clusters, sizes=sizes, noise=noise, aniso=aniso,
             metric=metric, method=method, precision=precision, doublets=doublets)
    return c if name is None else dict(c, name=name)


# ---- inputs -------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _mixture(n, d, clusters, seed, sizes=0.0, noise=0.0, aniso=False, normalize=False):
    g = _gen(seed)
    w = torch.exp(sizes * torch.randn(clusters, generator=g, device=DEV))
    centres = 5.0 * torch.randn((clusters, d), generator=g, device=DEV)
    lab = torch.multinomial(w / w.sum(), n, replacement=True, generator=g)
    X = torch.randn((n, d), generator=g, device=DEV)
    if aniso:
        X *= torch.exp(0.5 * torch.randn((clusters, d), generator=g, device=DEV))[lab]
    X += centres[lab]
    m = int(round(n * noise))
    if m:
        at = torch.randperm(n, generator=g, device=DEV)[:m]
        lo, hi = centres.amin(0), centres.amax(0)
        X[at] = lo + (hi - lo) * torch.rand((m, d), generator=g, device=DEV)
    if normalize:
        X = torch.nn.functional.normalize(X.double(), dim=1).float()
    return X.contiguous()


def _embedding(case, seed):
    if case["doublets"]:                 # a third observed, the rest midpoints of random pairs
        n = case["n"] // 3
        X = _mixture(n, case["d"], case["clusters"], seed)
        g = _gen(seed + 1)
        m = case["n"] - n
        a, b = torch.randint(0, n, (2, m), generator=g, device=DEV)
        sim = 0.5 * (X[a] + X[b]) + 0.05 * torch.randn((m, case["d"]), generator=g, device=DEV)
        return torch.cat([X, sim]).contiguous()
    return _mixture(case["n"], case["d"], case["clusters"], seed, case["sizes"], case["noise"],
                    case["aniso"], case["metric"] == "cosine")


def _cohort_sizes(case):
    r = np.random.default_rng(case["shape_seed"])
    return np.clip(np.round(r.lognormal(math.log(case["median"]), 0.9, case["samples"])),
                   2_000, 100_000).astype(np.int64)


def _cohort(case, seed):
    ns = _cohort_sizes(case)
    r = np.random.default_rng(case["shape_seed"] + 1)
    X = torch.cat([_mixture(int(n), case["d"], int(r.integers(10, 41)), seed * 1000 + s, 0.5)
                   for s, n in enumerate(ns)])
    return X, np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)


def _batches(case, seed):
    """Cells of every batch drawn from the same clusters, each batch shifted a little."""
    X = _mixture(case["n"], case["d"], case["clusters"], seed, 0.5)
    g = _gen(seed + 1)
    codes = torch.randint(0, case["batches"], (case["n"],), generator=g, device=DEV)
    X += torch.randn((case["batches"], case["d"]), generator=g, device=DEV)[codes]
    return X, codes.to(torch.int32)


def _regions():
    """Centres and spreads (µm) of a slide's 12 tissue regions on a 10 mm field."""
    r = np.random.default_rng(7)
    return r.uniform(1500, 8500, (12, 2)), r.uniform(300, 900, 12)


def _slide(case, seed):
    """Spots in µm on a 10 mm field: 70% in the tissue regions, 30% uniform background."""
    n, g = case["n"], _gen(seed)
    centres, sig = (torch.from_numpy(a).to(DEV) for a in _regions())
    lab = torch.randint(0, 12, (n,), generator=g, device=DEV)
    xy = centres[lab] + sig[lab, None] * torch.randn((n, 2), generator=g, device=DEV,
                                                     dtype=torch.float64)
    back = torch.rand(n, generator=g, device=DEV) < 0.3
    uni = 10_000 * torch.rand((n, 2), generator=g, device=DEV, dtype=torch.float64)
    return torch.where(back[:, None], uni, xy).float().contiguous()


def _spots_within(n, radius):
    """Expected number of (spot, other spot) pairs of a slide within a radius."""
    c, s = _regions()
    v = s[:, None] ** 2 + s[None, :] ** 2
    sep = ((c[:, None] - c[None, :]) ** 2).sum(2)
    tissue = (np.exp(-sep / (2 * v)) / (2 * math.pi * v)).mean()
    return math.pi * radius ** 2 * n * n * (0.49 * tissue + (0.42 + 0.09) * 1e-8)


def _fuzzy_graph(case, seed):
    """A symmetric graph in the layout of a graph result: about 2·(k-1) edges per cell, of cells
    in the same neighbourhood, weights between 0 and 1 as fuzzy unions have them (a fixed set of
    them, dealt out by the seed)."""
    n, k = case["n"], case["k"]
    m = n * (k - 1)
    i = torch.arange(n, device=DEV).repeat_interleave(k - 1)
    j = (i + torch.randint(1, 200, (m,), generator=_gen(11), device=DEV)) % n
    pair = torch.unique(torch.minimum(i, j) * n + torch.maximum(i, j))
    u = torch.randperm(pair.numel(), generator=_gen(seed), device=DEV).double() / pair.numel()
    w = torch.exp(-6.0 * u * u).float()
    i, j = pair // n, pair % n
    key, o = torch.sort(torch.cat([i * n + j, j * n + i]))
    w = torch.cat([w, w])[o]
    i, j = key // n, key % n
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(i, minlength=n), 0)
    return {"conn_indptr": ptr, "conn_indices": j.to(torch.int32), "conn_data": w}


def _room(case):
    m = _spots_within(case["n"], case["radius"])
    return int(1.05 * m + 20 * math.sqrt(m))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("graph", "knn"):
        s["X"], s["ws"] = _embedding(case, seed), nbm.Workspace(torch.device(DEV, 0))
        if kind == "graph":            # the result's buffers, kept from call to call
            m = 2 * case["n"] * (case["k"] - 1)
            s["out"] = {"conn_indices": torch.zeros(m, dtype=torch.int32, device=DEV),
                        "conn_data": torch.zeros(m, dtype=torch.float32, device=DEV)}
    elif kind == "host":
        s["X"] = _embedding(case, seed).cpu().pin_memory()
        s["buffers"] = nbm.HostGraphState(case["n"], case["d"], case["k"])
        for t in s["buffers"].host.values():
            t.zero_()
    elif kind == "cohort":
        s["X"], off = _cohort(case, seed)
        s["plan"] = mbatch.BatchedKnn(off, case["d"], case["k"])
    elif kind == "bbknn":
        s["X"], s["codes"] = _batches(case, seed)
        s["counts"] = torch.bincount(s["codes"], minlength=case["batches"]).cpu().numpy()
        s["ws"] = nbm.Workspace(torch.device(DEV, 0))
    elif kind == "umap_edges":
        s["graph"] = _fuzzy_graph(case, seed)
    else:
        s["X"], s["ws"] = _slide(case, seed), nbm.Workspace(torch.device(DEV, 0))
        if kind == "spatial_radius":
            s["room"] = _room(case)
    return s


# ---- one pass -----------------------------------------------------------------------------------

GRAPH = ("dist_indptr", "dist_indices", "dist_data", "conn_indptr", "conn_indices", "conn_data")


def _valid(ptr, a):
    """A buffer of a graph's largest size with zeros behind the entries it has."""
    return torch.where(torch.arange(a.numel(), device=a.device) < ptr[-1], a, 0)


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "graph":
        r = nbm.neighbors_device(s["X"], c["k"], metric=c["metric"], method=c["method"],
                                 precision=c["precision"], workspace=s["ws"], out=s["out"])
        return {k: r[k] for k in ("knn_idx", "knn_dist") + GRAPH}
    if kind == "host":
        r = nbm.neighbors_host(s["X"], c["k"], metric=c["metric"], method=c["method"],
                               precision=c["precision"], state=s["buffers"])
        return {k: r[k] for k in GRAPH}
    if kind == "knn":
        idx, dist, _ = nbm.knn_device(s["X"], c["k"], metric=c["metric"],
                                      precision=c["precision"], workspace=s["ws"])
        return {"knn_idx": idx, "knn_dist": dist}
    if kind == "cohort":
        idx, dist = s["plan"].run(s["X"])
        return {"knn_idx": idx, "knn_dist": dist}
    if kind == "bbknn":
        r = mbb.bbknn_device(s["X"], s["codes"], s["counts"], c["within"], workspace=s["ws"])
        out = {k: r[k] for k in ("knn_idx", "knn_dist", "dist_indptr", "conn_indptr")}
        for k in ("dist", "conn"):
            out.update({k + w: _valid(r[k + "_indptr"], r[k + w]) for w in ("_indices", "_data")})
        return out
    if kind == "spatial_knn":
        idx, dist, _ = msp.knn_grid_device(s["X"], c["k"], s["ws"])
        return {"idx": idx, "dist": dist}
    if kind == "spatial_radius":
        ptr, cols, dist, _ = msp.radius_grid_device(s["X"], c["radius"], 0.0, s["ws"])
        room = s["room"] - cols.numel()                 # the number of pairs depends on the data
        return {"indptr": ptr, "cols": torch.nn.functional.pad(cols, (0, room)),
                "dist": torch.nn.functional.pad(dist, (0, room))}
    e = nbm.umap_edges(s["graph"], c["n"])
    return {k: e[k] for k in ("indptr", "rows", "cols", "weights", "epochs_per_sample")}


def work(case):
    """Bytes: the inputs once, the outputs once.  Operations: the distances from every cell to
    the cells of its own cluster, which no exact search can leave out (2·d each); the spatial
    search: to the points of the 3×3 cells around it."""
    c, kind = case, case["kind"]
    if kind in ("graph", "host", "knn"):
        n, d, k = c["n"], c["d"], c["k"]
        own = n / c["clusters"] * math.exp(c["sizes"] ** 2)       # E[size²] / E[size]
        out = 8 * n * k
        if kind != "knn":
            out += 8 * n * (k - 1) + 16 * (n + 1) + 8 * 1.6 * n * (k - 1)
        return {"bytes": 4 * n * d + out, "flops": 2.0 * d * n * min(n, own)}
    if kind == "cohort":
        ns = _cohort_sizes(c).astype(float)
        return {"bytes": ns.sum() * (4 * c["d"] + 8 * c["k"]),
                "flops": 2.0 * c["d"] * float((ns ** 2).sum()) / 25 * math.exp(0.25)}
    if kind == "bbknn":
        n, K = c["n"], c["batches"] * c["within"]
        return {"bytes": n * (4 * c["d"] + 4 + 8 * K + 8 * (K - 1) + 16 + 1.6 * 8 * (K - 1)),
                "flops": 2.0 * c["d"] * n * n / c["clusters"] * math.exp(0.25)}
    if kind == "spatial_knn":
        return {"bytes": c["n"] * (8 + 8 * c["k"]), "flops": c["n"] * 9.0 * 2 * c["k"] * 5}
    if kind == "spatial_radius":
        m = _spots_within(c["n"], c["radius"])
        return {"bytes": 16.0 * c["n"] + 8 * m, "flops": m * 9 / math.pi * 5}
    nnz = 1.9 * c["n"] * (c["k"] - 1)
    return {"bytes": 8 * (c["n"] + 1) * 2 + nnz * 8 + 0.94 * nnz * 20, "flops": nnz}


# ---- the same in 64 bits ------------------------------------------------------------------------

def _knn64(Q, K, k, self_at=None):
    """(columns, squared distances) of every row of Q's k nearest rows of K, FP64, ascending;
    self_at: the row of K that a row of Q itself is (first in its list, at distance 0)."""
    sq = (K * K).sum(1)
    cols, d2s = [], []
    step = max(128, int(1.5e9 // max(K.shape[0], 1)) // 4)
    for a in range(0, Q.shape[0], step):
        q = Q[a:a + step]
        d2 = sq[None, :] - 2.0 * (q @ K.T)
        if self_at is not None:
            me = self_at[a:a + step]
            r = torch.nonzero(me >= 0).squeeze(1)
            d2[r, me[r]] = -math.inf
        m = min(K.shape[0], k + 8)
        c = torch.topk(d2, m, largest=False).indices
        del d2
        e = ((q[:, None, :] - K[c]) ** 2).sum(2)
        if self_at is not None:
            e = torch.where(c == self_at[a:a + step, None], -1.0, e)
        e, o = torch.sort(e, dim=1)
        cols.append(torch.gather(c, 1, o)[:, :k])
        d2s.append(e[:, :k].clamp_min(0.0))
    return torch.cat(cols), torch.cat(d2s)


def _smooth64(D, k):
    """umap's σ and ρ of every row (local connectivity 1), FP64."""
    n, kc = D.shape
    nz = D > 0
    first = torch.argmax(nz.int(), 1)
    rho = torch.where(nz.any(1), D[torch.arange(n, device=D.device), first], 0.0)
    lo, hi = torch.zeros_like(rho), torch.full_like(rho, math.inf)
    mid, live = torch.ones_like(rho), torch.ones(n, dtype=torch.bool, device=D.device)
    over = (D[:, 1:] - rho[:, None])
    for _ in range(64):
        s = torch.where(over > 0, torch.exp(-over / mid[:, None]), 1.0).sum(1)
        live &= (s - math.log2(k)).abs() >= 1e-5
        if not bool(live.any()):
            break
        up = live & (s > math.log2(k))
        dn = live & ~up
        hi = torch.where(up, mid, hi)
        lo = torch.where(dn, mid, lo)
        mid = torch.where(live, torch.where(torch.isinf(hi), mid * 2, (lo + hi) / 2), mid)
    floor = torch.where(rho > 0, D.mean(1), D.mean()) * 1e-3
    return torch.maximum(mid, floor), rho


def _union64(n, i, j, w):
    """a + b − a·b of both directions of every edge: (row, column, value), rows ascending."""
    keep = w.float() != 0                    # what float32 cannot hold is no edge of the matrix
    i, j, w = i[keep], j[keep], w[keep]
    key, inv = torch.unique(torch.cat([i * n + j, j * n + i]), return_inverse=True)
    a = torch.zeros(key.numel(), dtype=torch.float64, device=w.device)
    b = torch.zeros_like(a)
    a[inv[:i.numel()]] = w
    b[inv[i.numel():]] = w
    v = a + b - a * b
    return key // n, key % n, v


def _graph64(idx, dist, k, method):
    """(distances data, connectivities (row, column, value)) of the lists."""
    n = idx.shape[0]
    o = torch.argsort(idx[:, 1:], dim=1)
    dist_data = torch.gather(dist[:, 1:], 1, o).reshape(-1)
    rows = torch.arange(n, device=idx.device).repeat_interleave(idx.shape[1])
    if method == "umap":
        sigma, rho = _smooth64(dist, k)
        w = torch.where(dist <= rho[:, None], 1.0,
                        torch.exp(-(dist - rho[:, None]) / sigma[:, None]))
        w = torch.where(idx == torch.arange(n, device=idx.device)[:, None], 0.0, w)
        return dist_data, _union64(n, rows, idx.reshape(-1), w.reshape(-1))
    sq = dist[:, 1:] ** 2
    s = torch.sort(sq, dim=1).values
    m = s.shape[1]
    s2 = 0.5 * (s[:, (m - 1) // 2] + s[:, m // 2])
    rows = torch.arange(n, device=idx.device).repeat_interleave(m)
    c = idx[:, 1:].reshape(-1)
    key, inv = torch.unique(torch.cat([rows * n + c, c * n + rows]), return_inverse=True)
    d2 = torch.zeros(key.numel(), dtype=torch.float64, device=idx.device)
    d2[inv] = torch.cat([sq.reshape(-1)] * 2)
    i, j = key // n, key % n
    den = s2[i] + s2[j]
    return dist_data, (i, j, torch.sqrt(2 * torch.sqrt(s2[i] * s2[j]) / den) * torch.exp(-d2 / den))


def _near64(X, k=0, radius=0.0):
    """k nearest or all points within a radius, FP64 distances: the points in order of x, every
    chunk of queries against those in its band of x (widened until it holds every neighbour)."""
    n = X.shape[0]
    order = torch.argsort(X[:, 0])
    P = X[order].double()
    xs = P[:, 0].contiguous()
    got, step = [], 2048
    for a in range(0, n, step):
        q = P[a:a + step]
        m = q.shape[0]
        band = radius * 1.001 if radius else 60.0
        while True:
            b = int(torch.searchsorted(xs, q[0, 0] - band))
            e = int(torch.searchsorted(xs, q[-1, 0] + band, right=True))
            c = P[b:e]
            if radius:
                # which pairs are edges is decided in float32, as the matrix is defined
                qf, cf = q.float(), c.float()
                dx, dy = qf[:, None, 0] - cf[None, :, 0], qf[:, None, 1] - cf[None, :, 1]
                hit = dx * dx + dy * dy <= torch.tensor(radius * radius, device=X.device).float()
                hit[torch.arange(m), torch.arange(a - b, a - b + m)] = False
                r, t = torch.nonzero(hit, as_tuple=True)
                got.append((order[a + r], order[b + t], (q[r] - c[t]).square().sum(1).sqrt()))
                break
            d2 = (q[:, None, 0] - c[None, :, 0]) ** 2 + (q[:, None, 1] - c[None, :, 1]) ** 2
            if c.shape[0] >= k:
                v = torch.topk(d2, k, largest=False).values.sort(1).values.sqrt()
                if (b == 0 and e == n) or bool((v[:, -1] <= band).all()):
                    got.append((order[a:a + step], v))
                    break
            band *= 4
    return got


def exact(case, seed):
    kind = case["kind"]
    n = case.get("n", 0)
    if kind in ("graph", "host", "knn"):
        if n > 250_000:
            return None
        X = _embedding(case, seed).double()
        if case["metric"] == "cosine":
            X = torch.nn.functional.normalize(X, dim=1)
        idx, d2 = _knn64(X, X, case["k"], torch.arange(n, device=X.device))
        dist = d2 / 2 if case["metric"] == "cosine" else d2.sqrt()
        if kind == "knn":
            return {"knn_idx": None, "knn_dist": dist}
        dd, (_, _, v) = _graph64(idx, dist, case["k"], case["method"])
        v = torch.nn.functional.pad(v, (0, 2 * n * (case["k"] - 1) - v.numel()))
        out = {"dist_indptr": None, "dist_indices": None, "dist_data": dd, "conn_indptr": None,
               "conn_indices": None, "conn_data": v}
        return out if kind == "host" else dict(out, knn_idx=None, knn_dist=dist)
    if kind == "cohort":
        X, off = _cohort(case, seed)
        X = X.double()
        d2 = [_knn64(X[a:b], X[a:b], case["k"], torch.arange(b - a, device=X.device))[1]
              for a, b in zip(off[:-1], off[1:])]
        return {"knn_idx": None, "knn_dist": torch.cat(d2).sqrt()}
    if kind == "bbknn":
        X, codes = _batches(case, seed)
        X = X.double()
        me = torch.arange(n, device=X.device)
        cols, d2s = [], []
        for b in range(case["batches"]):
            rows = torch.nonzero(codes == b).squeeze(1)
            where = torch.full((n,), -1, dtype=torch.int64, device=X.device)
            where[rows] = torch.arange(rows.numel(), device=X.device)
            c, d2 = _knn64(X, X[rows], min(case["within"], rows.numel()), where)
            cols.append(rows[c])
            d2s.append(d2)
        d2, o = torch.sort(torch.cat(d2s, 1), dim=1, stable=True)
        idx, dist = torch.gather(torch.cat(cols, 1), 1, o), d2.sqrt()
        K = idx.shape[1]
        sigma, rho = _smooth64(dist, K)
        w = torch.where(dist <= rho[:, None], 1.0,
                        torch.exp(-(dist - rho[:, None]) / sigma[:, None]))
        w = torch.where(idx == me[:, None], 0.0, w)
        i, j, v = _union64(n, me.repeat_interleave(K), idx.reshape(-1), w.reshape(-1))
        # trimmed to the 10·K strongest of either end
        by = torch.argsort(v, descending=True, stable=True)
        by = by[torch.argsort(i[by], stable=True)]
        cnt = torch.bincount(i, minlength=n)
        start = torch.cumsum(cnt, 0) - cnt
        long = cnt > 10 * K
        theta = torch.full((n,), -math.inf, dtype=torch.float64, device=X.device)
        theta[long] = v[by[start[long] + 10 * K - 1]]
        v = v[(v >= theta[i]) & (v >= theta[j])]
        o = torch.argsort(idx, dim=1)
        dd = torch.gather(dist, 1, o)
        dd = dd[(torch.gather(idx, 1, o) != me[:, None]) & (dd > 0)]
        dd = torch.nn.functional.pad(dd, (0, n * K - dd.numel()))
        v = torch.nn.functional.pad(v, (0, 2 * n * K - v.numel()))
        return {"knn_idx": None, "knn_dist": dist, "dist_indptr": None, "dist_indices": None,
                "dist_data": dd, "conn_indptr": None, "conn_indices": None, "conn_data": v}
    if kind == "spatial_knn":
        out = torch.empty((n, case["k"]), dtype=torch.float64, device=DEV)
        for rows, v in _near64(_slide(case, seed), k=case["k"]):
            out[rows] = v
        return {"idx": None, "dist": out}
    if kind == "spatial_radius":
        got = _near64(_slide(case, seed), radius=case["radius"])
        i, j, v = (torch.cat([g[t] for g in got]) for t in range(3))
        v = torch.nn.functional.pad(v[torch.argsort(i * n + j)], (0, _room(case) - v.numel()))
        return {"indptr": None, "cols": None, "dist": v}
    g = _fuzzy_graph(case, seed)
    w = g["conn_data"].double()
    epochs = 500 if n <= 10_000 else 200
    w = w[w >= w.max() / epochs]
    return {"indptr": None, "rows": None, "cols": None, "weights": w,
            "epochs_per_sample": w.max() / w}
