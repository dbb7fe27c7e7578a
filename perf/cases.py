"""The workloads that HDBSCAN's speed is measured on: what each takes in, one
pass of it through the public entry points, and the bytes and operations that
pass cannot do without.

A case is a dict of plain values.  `kind` selects the entry point:

  fit          HDBSCAN(...).fit(X), the fitted attributes returned
  labels       fast_hdbscan(X, ...), labels and probabilities only
  weighted     HDBSCAN(...).fit(X, sample_weight=w)
  precomputed  fhg_hdbscan_fit_precomputed on a kNN distance graph (COO)
  batch        batch.fit_many on many uneven instances

The sizes are those of the synthetic benchmark workloads (20,000 x 2,
2,000,000 x 5, 10,000,000 x 3, x 64, a kNN-graph Kruskal, a precomputed kNN
graph, uneven batches) or of the tests, with odd and ragged ones among them.
"""
import ctypes
import math

import numpy as np
import torch

from fast_hdbscan_gb300 import HDBSCAN, _native, fast_hdbscan
from fast_hdbscan_gb300.batch import fit_many
from fast_hdbscan_gb300.numba_kdtree import build_kdtree, parallel_tree_query

_BASE = {"kind": "fit", "data": "blobs", "n": 0, "d": 2, "ms": 10, "mcs": 50, "host": False,
         "method": "eom", "algorithm": "boruvka", "knn_k": 0, "reproducible": False, "count": 1}


# Estimator cases of up to this many points return the condensed tree too.
_TREE_ROWS = 20_000


def _case(**kw):
    c = dict(_BASE)
    c.update(kw)
    return c


def listed():
    return [
        # a notebook call with the defaults: a few hundred points, latency only
        _case(name="tiny_defaults", n=397, d=2, ms=0, mcs=5, host=True),
        # the small benchmark workload, a NumPy array in, the attributes out
        _case(name="blobs_20k_2d", n=20_000, d=2, ms=10, mcs=50, host=True),
        # a UMAP-like embedding already on the GPU, the attributes out
        _case(name="umap_2m_5d", n=2_000_000, d=5, ms=10, mcs=500),
        # the headline workload: widely varying density, labels wanted
        _case(name="density_10m_3d", kind="labels", data="density", n=10_000_000, d=3, ms=15,
              mcs=500),
        # an embedding of more than eight dimensions, ragged size, leaf clusters
        _case(name="embedding_60k_13d", kind="labels", n=60_013, d=13, ms=10, mcs=100,
              method="leaf"),
        # min_cluster_size alone: min_samples follows it, lists of 101 neighbours
        _case(name="mcs100_300k_3d", data="density", n=300_001, d=3, ms=0, mcs=100),
        # more than 30 dimensions: the exact kNN-graph route
        _case(name="highd_150k_64d", data="aniso", n=150_000, d=64, ms=10, mcs=500),
        # algorithm="kruskal" on the spatial index's kNN graph
        _case(name="kruskal_1m_3d", data="density", n=1_000_003, d=3, ms=15, mcs=500,
              algorithm="kruskal", knn_k=16),
        # metric="precomputed": a 15-nearest-neighbour distance graph
        _case(name="precomputed_300k", kind="precomputed", data="density", n=300_000, d=3, ms=10,
              mcs=100, knn_k=15, algorithm="kruskal"),
        # many uneven clusterings in one call
        _case(name="batch_192", kind="batch", n=20_000, d=0, count=192),
        # the reference's own tie choices
        _case(name="reproducible_1m_2d", n=1_000_000, d=2, ms=5, mcs=200, reproducible=True),
        # sample weights
        _case(name="weighted_200k_4d", kind="weighted", n=200_003, d=4, ms=10, mcs=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["fit", "fit", "labels", "labels", "wide", "long", "highd", "kruskal",
                       "precomputed", "batch", "reproducible", "weighted"])
    data = rng.choice(["blobs", "density"])
    method = rng.choice(["eom", "eom", "leaf"])
    ms = rng.choice([3, 5, 7, 10, 15, 20])
    if what in ("fit", "labels"):
        n = _log_int(rng, 200, 4_000_000)
        return _case(kind=what, data=data, n=n, d=rng.randint(1, 6), ms=ms,
                     mcs=max(5, min(500, n // 100)), method=method, host=n < 100_000)
    if what == "wide":
        d = rng.randint(7, 24)
        n = _log_int(rng, 2_000, 60_000)
        return _case(kind="labels", n=n, d=d, ms=ms, mcs=max(10, n // 500), method=method)
    if what == "long":
        mcs = rng.randint(64, 250)
        return _case(data=data, n=_log_int(rng, 2_000, 300_000), d=rng.randint(2, 4), ms=0,
                     mcs=mcs, method=method)
    if what == "highd":
        n = _log_int(rng, 2_000, 150_000)
        return _case(data="aniso", n=n, d=rng.randint(31, 64), ms=rng.choice([5, 10]),
                     mcs=max(10, n // 300))
    if what == "kruskal":
        n = _log_int(rng, 5_000, 2_000_000)
        return _case(data=data, n=n, d=rng.randint(2, 5), ms=ms, mcs=max(10, min(500, n // 100)),
                     algorithm="kruskal", knn_k=rng.randint(10, 30))
    if what == "precomputed":
        n = _log_int(rng, 2_000, 500_000)
        return _case(kind="precomputed", data=data, n=n, d=rng.randint(2, 5),
                     ms=rng.choice([5, 10]), mcs=max(10, n // 1000), knn_k=rng.randint(10, 20),
                     algorithm=rng.choice(["boruvka", "kruskal"]))
    if what == "batch":
        return _case(kind="batch", n=_log_int(rng, 1_000, 40_000), d=0,
                     count=_log_int(rng, 16, 192))
    n = _log_int(rng, 1_000, 500_000)
    if what == "reproducible":
        return _case(data=data, n=n, d=rng.randint(2, 4), ms=ms, mcs=max(10, min(200, n // 100)),
                     reproducible=True, method=method)
    return _case(kind="weighted", data=data, n=n, d=rng.randint(2, 5), ms=ms,
                 mcs=max(10, min(100, n // 100)))


# ------------------------------------------------------------------- inputs
def _points(case, seed):
    """n x d float32 points on the GPU, from the seed alone: "blobs" = 40
    Gaussian blobs of unequal weight and spread with uniform noise, "density"
    = 200 Gaussians of widely varying spread, "aniso" = anisotropic
    Gaussians."""
    n, d = case["n"], case["d"]
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (seed + 1) + n + 31 * d)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    def uniform(*shape):
        return torch.rand(*shape, generator=g, device="cuda")

    if case["data"] == "aniso":
        comp = 50 if n >= 20_000 else 10
        which = torch.sort(torch.randint(0, comp, (n,), generator=g, device="cuda"))[0]
        counts = torch.bincount(which, minlength=comp).tolist()
        centers, spread = 2.0 * normal(comp, d), 0.3 * normal(comp, d, d)
        parts = [centers[c] + normal(m, d) @ spread[c].T for c, m in enumerate(counts)]
        x = torch.cat(parts)
    elif case["data"] == "density":
        comp = 200 if n >= 20_000 else 20
        centers = 200.0 * uniform(comp, d) - 100.0
        stds = torch.exp(normal(comp))
        which = torch.randint(0, comp, (n,), generator=g, device="cuda")
        x = centers[which] + normal(n, d) * stds[which, None]
    else:
        comp = 40 if n >= 20_000 else 8
        noise = n // 10
        centers = 40.0 * uniform(comp, d) - 20.0
        stds = torch.exp(math.log(0.2) + uniform(comp) * math.log(10.0))
        weights = -torch.log(uniform(comp).clamp_min(1e-6))
        which = torch.multinomial(weights, n - noise, replacement=True, generator=g)
        pts = centers[which] + normal(n - noise, d) * stds[which, None]
        lo, hi = pts.min(0).values, pts.max(0).values
        x = torch.cat([pts, lo + uniform(noise, d) * (hi - lo)])
    x = x[torch.randperm(n, generator=g, device="cuda")]
    return x.to(torch.float32).contiguous()


def _instances(case, seed):
    """Uneven mixtures, n log-uniform in [200, case n], d in 2..8, with 5 %
    noise: NumPy arrays, as a caller of fit_many holds them.  The sizes
    belong to the case, the points to the seed."""
    sizes = np.random.default_rng(case["count"] + case["n"])
    rng = np.random.default_rng(seed + 17)
    out, ms, mcs = [], [], []
    for _ in range(case["count"]):
        n = int(np.exp(sizes.uniform(np.log(200), np.log(case["n"]))))
        d, k = int(sizes.integers(2, 9)), int(rng.integers(3, 13))
        centers = rng.uniform(-10.0, 10.0, size=(k, d))
        x = centers[rng.integers(0, k, size=n)] + rng.normal(size=(n, d))
        m = n // 20
        x[:m] = rng.uniform(x.min(axis=0), x.max(axis=0), size=(m, d))
        out.append(np.ascontiguousarray(x[rng.permutation(n)], dtype=np.float32))
        ms.append(int(rng.choice([5, 10, 20])))
        mcs.append(max(10, n // 100))
    return out, ms, mcs


def _knn_graph(case, seed):
    """The k-nearest-neighbour distance graph of the points, row by row."""
    x = _points(case, seed)
    dist, idx = parallel_tree_query(*_tree(x), k=case["knn_k"] + 1)
    n, k = dist.shape
    rows = torch.arange(n, dtype=torch.int32, device="cuda").repeat_interleave(k - 1)
    cols = torch.from_numpy(idx[:, 1:].astype(np.int32)).cuda().reshape(-1).contiguous()
    data = torch.from_numpy(dist[:, 1:].astype(np.float64)).cuda().reshape(-1).contiguous()
    return rows, cols, data


def _tree(x):
    tree = build_kdtree(x.cpu().numpy())
    return tree, tree.data


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "batch":
        state["instances"], state["ms"], state["mcs"] = _instances(case, seed)
    elif kind == "precomputed":
        state["graph"] = _knn_graph(case, seed)
    else:
        x = _points(case, seed)
        if kind == "weighted":
            # class weights of 1 to 4, in equal parts
            w = (np.arange(case["n"]) % 4 + 1).astype(np.float32)
            state["weights"] = np.random.default_rng(seed).permutation(w)
            case = dict(case, host=True)  # weights go with host points
        state["x"] = x.cpu().numpy() if case["host"] else x
    return state


# --------------------------------------------------------------------- pass
def _fit_precomputed(case, graph):
    """metric="precomputed" through the C entry point, device to device."""
    rows, cols, data = graph
    n, ms = case["n"], case["ms"]

    def empty(*shape, dtype):
        return torch.empty(*shape, dtype=dtype, device="cuda")

    i64, f32, f64 = torch.int64, torch.float32, torch.float64
    labels, probs, sel = empty(n, dtype=i64), empty(n, dtype=f32), empty(n, dtype=i64)
    mst, linkage = empty(n - 1, 3, dtype=f64), empty(n - 1, 4, dtype=f64)
    parent, child = empty(2 * n, dtype=i64), empty(2 * n, dtype=i64)
    lam, size = empty(2 * n, dtype=f32), empty(2 * n, dtype=f32)
    nbrs, core = empty(n, ms, dtype=torch.int32), empty(n, dtype=f64)
    n_rows, n_sel = ctypes.c_int64(0), ctypes.c_int64(0)
    p = _native.vptr
    _native.check(_native.load().fhg_hdbscan_fit_precomputed(
        p(rows), p(cols), p(data), data.numel(), n, ms, int(case["algorithm"] == "kruskal"),
        case["mcs"], 0, math.inf, 0, 0.0, 0.0, p(labels), p(probs), p(mst), p(linkage),
        p(parent), p(child), p(lam), p(size), ctypes.byref(n_rows), p(nbrs), p(core), p(sel),
        ctypes.byref(n_sel), _native.stream_ptr()))
    for rows_of in (parent, child, lam, size):  # the room past the last row
        rows_of[n_rows.value:] = 0
    return {"labels": labels, "probabilities": probs, "mst": mst, "linkage": linkage,
            "parent": parent, "child": child, "lambda_val": lam, "child_size": size,
            "neighbors": nbrs, "core": core}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        res = fit_many(state["instances"], state["ms"], state["mcs"])
        return {"labels": np.concatenate([a for a, _ in res]),
                "probabilities": np.concatenate([b for _, b in res])}
    if case["kind"] == "precomputed":
        return _fit_precomputed(case, state["graph"])
    options = dict(min_samples=case["ms"] or None, min_cluster_size=case["mcs"],
                   cluster_selection_method=case["method"], algorithm=case["algorithm"],
                   knn_k=case["knn_k"] or None, reproducible=case["reproducible"])
    if case["kind"] == "labels":
        labels, probs = fast_hdbscan(state["x"], **options)
        return {"labels": labels, "probabilities": probs}
    m = HDBSCAN(**options).fit(state["x"], sample_weight=state.get("weights"))
    out = {"labels": m.labels_, "probabilities": m.probabilities_,
           "linkage": m._single_linkage_tree, "mst": m._min_spanning_tree,
           "neighbors": m._neighbors, "core": m._core_distances}
    if case["n"] <= _TREE_ROWS:
        # as many rows as its clusters ask for: at the room it can take, 2 n,
        # where copying it there is small beside the pass
        tree = m._condensed_tree
        for name in ("parent", "child", "lambda_val", "child_size"):
            out[name] = np.zeros(2 * case["n"], dtype=tree.dtype[name])
            out[name][:len(tree)] = tree[name]
    return out


# --------------------------------------------------------------------- work
def _list_len(case):
    ms = case["ms"] or case["mcs"]
    if case["kind"] == "weighted":
        return max(2, int(2 * ms / 2.5))
    if case["d"] > 30:
        return max(3 * ms, 15) + 1
    return max(case["knn_k"], ms) + 1


def work(case):
    """Input read once and outputs written once (labels, probabilities and,
    from the estimator, MST, linkage tree, condensed tree, neighbours and core
    distances); the distances of every kNN
    list entry (3 d operations each), or every pair's inner product on the
    route that has no spatial index (more than 30 dimensions)."""
    n, d, k = case["n"], case["d"], _list_len(case)
    if case["kind"] == "batch":
        mean = (case["n"] - 200) / math.log(case["n"] / 200)
        pts = case["count"] * mean
        return {"bytes": pts * (4 * 5 + 12), "flops": pts * 12 * 15}
    if case["kind"] == "precomputed":
        nnz = n * case["knn_k"]
        return {"bytes": nnz * 16 + n * (12 + 56 + 24 * 1.2 + 4 * case["ms"] + 8),
                "flops": nnz}
    flops = 2.0 * n * n * d if d > 30 else 3.0 * n * k * d
    out = 12 if case["kind"] == "labels" else 12 + 24 + 32 + 28 * 1.2 + 4 * (k - 1) + 4
    return {"bytes": n * (4 * d + out), "flops": flops}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """The core distances in 64 bits, by brute force, where the points are few
    enough; every other output is whole or follows from order and ties."""
    if case["kind"] != "fit" or case["n"] > 150_000:
        return None
    x = _points(case, seed).double()
    n = case["n"]
    k = (case["ms"] or case["mcs"]) + 1  # the point itself included
    core = torch.empty(n, dtype=torch.float64, device="cuda")
    step = max(1, 100_000_000 // n)
    sq = (x * x).sum(1)
    for a in range(0, n, step):
        q = x[a:a + step]
        if case["d"] > 30:  # centred inputs: cancellation is far below float32
            d2 = (sq[a:a + step, None] + sq[None, :] - 2.0 * (q @ x.T)).clamp_min(0.0)
        else:
            d2 = torch.zeros(q.shape[0], n, dtype=torch.float64, device="cuda")
            for j in range(case["d"]):
                d2 += (q[:, j, None] - x[None, :, j]) ** 2
        core[a:a + step] = torch.topk(d2, min(k, n), dim=1, largest=False)[0][:, -1].sqrt()
    names = ["labels", "probabilities", "linkage", "mst", "neighbors"]
    if n <= _TREE_ROWS:
        names += ["parent", "child", "lambda_val", "child_size"]
    out = {name: None for name in names}
    out["core"] = core
    return out
