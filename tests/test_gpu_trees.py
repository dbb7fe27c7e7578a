"""GPU parity of the tree passes, fed the reference's own intermediates.

Every stage takes the reference's input from the fixtures (its raw MST, its
linkage tree, its condensed tree), so tie-breaking in the MST cannot enter:
sort, linkage tree, condensed tree, EOM / leaf selection, labels and
membership strengths must equal the reference's arrays exactly.
"""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

CASES = ["ka150", "blobs200", "blobs200_ms1", "blobs200_leaf", "blobs200_maxcs",
         "blobs200_single", "blobs2d_2k", "blobs2d_20k", "umap5d_5k", "vd3d_5k", "vd3d_20k",
         "edge_two", "edge_1d", "edge_highms", "edge_dups"]


def _golden(name):
    return np.load(os.path.join(GOLDEN, name + ".npz"))


def _ct(g):
    from fast_hdbscan_gb300.cluster_trees import CondensedTree

    return CondensedTree(g["ct_parent"], g["ct_child"], g["ct_lambda"], g["ct_size"])


@pytest.mark.parametrize("name", CASES)
def test_sort_and_linkage_bitexact(engine, name):
    from fast_hdbscan_gb300.cluster_trees import mst_to_linkage_tree, sort_mst

    g = _golden(name)
    smst = sort_mst(g["mst_raw"])
    np.testing.assert_array_equal(smst, g["sorted_mst"])
    np.testing.assert_array_equal(mst_to_linkage_tree(g["sorted_mst"]), g["linkage"])


@pytest.mark.parametrize("name", CASES)
def test_condense_bitexact(engine, name):
    from fast_hdbscan_gb300.cluster_trees import condense_tree

    g = _golden(name)
    # hdbscan.py:521 condenses without max_cluster_size (only EOM reads it)
    ct = condense_tree(g["linkage"], int(g["min_cluster_size"]))
    ref = _ct(g)
    for a, b in zip(ct, ref):
        np.testing.assert_array_equal(a, b)
        assert a.dtype == b.dtype


@pytest.mark.parametrize("name", CASES)
def test_selection_labels_bitexact(engine, name):
    from fast_hdbscan_gb300.cluster_trees import (
        cluster_tree_from_condensed_tree, cluster_tree_leaves, extract_eom_clusters,
        get_cluster_label_vector, get_point_membership_strength_vector)

    g = _golden(name)
    if str(g["cluster_selection_method"]) == "eom" and float(g["cluster_selection_epsilon"]) > 0:
        pytest.skip("epsilon search is checked elsewhere")
    if float(g["cluster_selection_persistence"]) > 0:
        pytest.skip("persistence is checked elsewhere")
    ct = _ct(g)
    n = g["X"].shape[0]
    cl_tree = cluster_tree_from_condensed_tree(ct)
    if str(g["cluster_selection_method"]) == "leaf":
        sel = cluster_tree_leaves(cl_tree, n) if len(cl_tree.parent) else np.empty(0, np.int64)
    else:
        sel = extract_eom_clusters(ct, cl_tree, float(g["max_cluster_size"]),
                                   bool(g["allow_single_cluster"]))
        if "selected_eom" in g.files:
            np.testing.assert_array_equal(sel, g["selected_eom"])
    labels = get_cluster_label_vector(ct, sel, 0.0, n)
    np.testing.assert_array_equal(labels, g["labels"])
    probs = get_point_membership_strength_vector(ct, sel, labels)
    np.testing.assert_array_equal(probs, g["probabilities"])


WEIGHTED = ["blobs200_w_labels", "blobs2d_2k_w", "vd3d_5k_w"]


@pytest.mark.parametrize("name", WEIGHTED)
def test_weighted_linkage_and_condense_bitexact(engine, name):
    """cluster_trees.py:98 mst_to_linkage_tree_w_sample_weights and :205
    condense_tree(sample_weights=...) on the reference's own sorted MST and
    linkage tree.  The fixtures' weights (integers, multiples of 1/64) have
    exact float32 sums, so the weighted sizes are bit-identical."""
    from fast_hdbscan_gb300.cluster_trees import (
        condense_tree, mst_to_linkage_tree_w_sample_weights, sort_mst)

    g = _golden(name)
    w = g["sample_weights"]
    np.testing.assert_array_equal(sort_mst(g["mst_raw"]), g["sorted_mst"])
    np.testing.assert_array_equal(mst_to_linkage_tree_w_sample_weights(g["sorted_mst"], w),
                                  g["linkage"])
    ct = condense_tree(g["linkage"], int(g["min_cluster_size"]), sample_weights=w)
    for a, b in zip(ct, _ct(g)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("name", CASES + WEIGHTED)
def test_clusters_from_spanning_tree_fused_bitexact(engine, name):
    """hdbscan.py:497 clusters_from_spanning_tree in one fused call
    (fhg_clusters_from_mst) on the reference's raw MST with the fixture's
    selection options: labels, probabilities, linkage tree, condensed tree and
    sorted MST equal the reference's arrays."""
    from fast_hdbscan_gb300.hdbscan import clusters_from_spanning_tree

    g = _golden(name)
    w = g["sample_weights"] if "sample_weights" in g.files else None
    labels, probs, linkage, ct, smst = clusters_from_spanning_tree(
        g["mst_raw"], min_cluster_size=int(g["min_cluster_size"]),
        cluster_selection_method=str(g["cluster_selection_method"]),
        max_cluster_size=float(g["max_cluster_size"]),
        allow_single_cluster=bool(g["allow_single_cluster"]),
        cluster_selection_epsilon=float(g["cluster_selection_epsilon"]),
        cluster_selection_persistence=float(g["cluster_selection_persistence"]),
        sample_weights=w)
    np.testing.assert_array_equal(smst, g["sorted_mst"])
    np.testing.assert_array_equal(linkage, g["linkage"])
    for a, b in zip(ct, _ct(g)):
        np.testing.assert_array_equal(a, b)
        assert a.dtype == b.dtype
    np.testing.assert_array_equal(labels, g["labels"])
    np.testing.assert_array_equal(probs, g["probabilities"])


@pytest.mark.parametrize("seed", range(6))
def test_clusters_from_spanning_tree_fused_vs_oracle(engine, seed):
    """The fused call against the oracle's clusters_from_spanning_tree on
    random trees with heavily tied integer weights (the sort's (weight, src,
    dst) order decides), both selection methods, epsilon, persistence,
    max_cluster_size, allow_single_cluster and sample weights."""
    from fast_hdbscan_gb300.hdbscan import clusters_from_spanning_tree
    from oracle import oracle as O

    rng = np.random.default_rng(seed)
    n = int(rng.integers(50, 3000))
    parent = np.array([rng.integers(0, i) for i in range(1, n)])
    child = np.arange(1, n)
    flip = rng.random(n - 1) < 0.5
    src, dst = np.where(flip, child, parent), np.where(flip, parent, child)
    wts = rng.integers(1, 12, size=n - 1).astype(np.float64) * 0.25
    mst = np.stack([src, dst, wts], axis=1).astype(np.float64)[rng.permutation(n - 1)]
    kw = dict(min_cluster_size=int(rng.integers(3, 40)),
              cluster_selection_method=["eom", "leaf"][seed % 2],
              max_cluster_size=[np.inf, float(n // 3)][(seed // 2) % 2],
              allow_single_cluster=bool(seed % 3 == 0),
              cluster_selection_epsilon=[0.0, 0.6][seed % 3 == 1],
              cluster_selection_persistence=[0.0, 0.3][seed % 4 == 2])
    w = (rng.integers(1, 5, size=n).astype(np.float32) if seed >= 4 else None)
    labels, probs, linkage, ct, smst = clusters_from_spanning_tree(mst, sample_weights=w, **kw)
    o_labels, o_probs, o_linkage, o_ct, o_smst, _ = O.clusters_from_spanning_tree(
        mst, sample_weights=w, **kw)
    np.testing.assert_array_equal(smst, o_smst)
    np.testing.assert_array_equal(linkage, o_linkage)
    for a, b in zip(ct, o_ct):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(labels, o_labels)
    np.testing.assert_array_equal(probs, o_probs)


def test_clusters_from_spanning_tree_weight_shape(engine):
    """A tree of m edges takes m + 1 sample weights; others are rejected
    before any device work."""
    from fast_hdbscan_gb300.hdbscan import clusters_from_spanning_tree

    mst = np.array([[0, 1, 0.5], [1, 2, 0.7], [2, 3, 0.2]])
    with pytest.raises(ValueError):
        clusters_from_spanning_tree(mst, min_cluster_size=2,
                                    sample_weights=np.ones(3, np.float32))
    labels, probs, *_ = clusters_from_spanning_tree(mst, min_cluster_size=2,
                                                    sample_weights=np.ones(4, np.float32))
    assert labels.shape == (4,) and probs.shape == (4,)


@pytest.mark.parametrize("C", [2, 33, 4095, 4096, 4097])
@pytest.mark.parametrize("shape", ["bushy", "chain"])
@pytest.mark.parametrize("big", [2047, 2048, 8192])
def test_eom_cluster_counts_vs_oracle(engine, C, shape, big):
    """Cluster trees on both sides of what the EOM kernel keeps in shared
    memory, wide and as deep as they have clusters, with clusters of 0 to 40
    rows and one on either side of the rows that a warp sums."""
    from fast_hdbscan_gb300.cluster_trees import (
        CondensedTree, cluster_tree_from_condensed_tree, extract_eom_clusters)
    from oracle import oracle as O

    rng = np.random.default_rng(C + big)
    lens = rng.integers(0, 41, size=C)
    lens[0] = max(lens[0], 1)
    lens[C // 2] = big
    n = int(lens.sum())
    up = np.maximum(np.arange(1, C) - 1, 0) if shape == "chain" else (
        rng.random(C - 1) * np.arange(1, C)).astype(np.int64)
    parent = np.concatenate([n + np.repeat(np.arange(C), lens), n + up])
    child = np.concatenate([np.arange(n), n + np.arange(1, C)])
    lam = (rng.random(n + C - 1) * 10).astype(np.float32)
    size = np.concatenate([np.ones(n), rng.integers(2, 1000, size=C - 1)]).astype(np.float32)
    # as in any condensed tree, a cluster's row comes before the rows under it
    order = np.concatenate([n + np.arange(C - 1), rng.permutation(n)])
    ct = CondensedTree(*[np.ascontiguousarray(a[order]) for a in (
        parent.astype(np.int64), child.astype(np.int64), lam, size)])
    for max_size in (np.inf, 500.0):
        for single in (False, True):
            sel = extract_eom_clusters(ct, cluster_tree_from_condensed_tree(ct), max_size, single)
            np.testing.assert_array_equal(sel, O.extract_eom_clusters(ct, max_size, single))


@pytest.mark.parametrize("m", [1, 511, 512, 513, 1024, 1025, 2049, 4096, 4097, 8193, 70_001])
@pytest.mark.parametrize("shape", ["random", "chain", "star", "pairs"])
def test_linkage_intervals_vs_oracle(engine, m, shape):
    """Edge counts around the intervals that one thread and one block take, on
    spanning trees with long chains, one hub, and many components to the end."""
    from fast_hdbscan_gb300.cluster_trees import mst_to_linkage_tree
    from oracle import oracle as O

    rng = np.random.default_rng(m)
    child = np.arange(1, m + 1)
    parent = {"random": (rng.random(m) * child).astype(np.int64), "chain": child - 1,
              "star": np.zeros(m, np.int64), "pairs": np.where(child % 2 == 1, child - 1,
                                                               child // 4)}[shape]
    w = rng.random(m) + (child % 2 == 0 if shape == "pairs" else 0)
    relabel = rng.permutation(m + 1)
    mst = np.stack([relabel[parent], relabel[child], w], axis=1).astype(np.float64)
    mst = mst[np.argsort(w, kind="stable")]
    np.testing.assert_array_equal(mst_to_linkage_tree(mst), O.mst_to_linkage_tree(mst))


@pytest.mark.parametrize("kind", ["weights", "random", "root", "zero", "large"])
@pytest.mark.parametrize("n", [40, 3000, 20_000])
@pytest.mark.parametrize("mcs", [2, 5, 40, 600])
def test_condense_sizes_that_are_no_counts(engine, kind, n, mcs):
    """A linkage tree whose size column is not the number of leaves (weight
    sums condensed without their weights, among others): the cases go by it,
    the rows by the points that there are, as in the reference."""
    from fast_hdbscan_gb300.cluster_trees import condense_tree
    from oracle import oracle as O

    rng = np.random.default_rng(n + mcs)
    child = np.arange(1, n)
    parent = np.where(rng.random(n - 1) < 0.5, child - 1, (rng.random(n - 1) * child).astype(int))
    w = np.sort(rng.integers(1, n, size=n - 1).astype(np.float64))
    mst = np.stack([parent, child, rng.permutation(w)], axis=1).astype(np.float64)
    weights = rng.integers(1, 5, size=n).astype(np.float32)
    linkage = O.mst_to_linkage_tree(O.sort_mst(mst), weights if kind == "weights" else None)
    size = linkage[:, 3]
    linkage[:, 3] = {"weights": size, "random": size * rng.integers(1, 4, size=n - 1),
                     "root": np.where(np.arange(n - 1) == n - 2, 3, size),
                     "zero": 0 * size, "large": size + 1000}[kind]
    got, expect = condense_tree(linkage, min_cluster_size=mcs), O.condense_tree(linkage, mcs)
    for a, b in zip(got, expect):
        np.testing.assert_array_equal(a, b)


def _cluster_tree(C, rng, big=0):
    """A condensed tree of C clusters of 0 to 100 rows, one of `big`, every
    cluster's row before the rows under it."""
    from fast_hdbscan_gb300.cluster_trees import CondensedTree

    lens = rng.integers(0, rng.integers(1, 101, size=C))
    lens[0] += 1
    lens[C // 3] += big
    n = int(lens.sum())
    up = (rng.random(C - 1) * np.arange(1, C)).astype(np.int64)
    parent = np.concatenate([n + up, n + np.repeat(np.arange(C), lens)])
    child = np.concatenate([n + np.arange(1, C), rng.permutation(n)])
    lam = (rng.random(n + C - 1) * 10).astype(np.float32)
    size = np.concatenate([rng.integers(2, 1000, size=C - 1), np.ones(n)]).astype(np.float32)
    return CondensedTree(parent.astype(np.int64), child.astype(np.int64), lam, size), n


@pytest.mark.parametrize("C", [16_384, 16_385, 40_000, 300_000])
@pytest.mark.parametrize("big", [0, 2047, 9000])
def test_eom_of_many_clusters_vs_oracle(engine, C, big):
    """A warp to a cluster's sum, and a lane or a warp each for 32 clusters."""
    from fast_hdbscan_gb300.cluster_trees import (
        cluster_tree_from_condensed_tree, extract_eom_clusters)
    from oracle import oracle as O

    ct, _ = _cluster_tree(C, np.random.default_rng(C + big), big)
    sel = extract_eom_clusters(ct, cluster_tree_from_condensed_tree(ct))
    np.testing.assert_array_equal(sel, O.extract_eom_clusters(ct))


@pytest.mark.parametrize("C", [16_384, 16_385, 300_000])
def test_labels_of_many_clusters_vs_oracle(engine, C):
    """Nearest selected clusters by one block and by launches."""
    from fast_hdbscan_gb300.cluster_trees import (
        get_cluster_label_vector, get_point_membership_strength_vector)
    from oracle import oracle as O

    rng = np.random.default_rng(C)
    ct, n = _cluster_tree(C, rng)
    clusters = n + np.sort(rng.choice(np.arange(1, C), C // 3, replace=False))
    labels = get_cluster_label_vector(ct, clusters, 0.0, n)
    np.testing.assert_array_equal(labels, O.get_cluster_label_vector(ct, clusters, 0.0, n))
    probs = get_point_membership_strength_vector(ct, clusters, labels)
    np.testing.assert_array_equal(
        probs, O.get_point_membership_strength_vector(ct, clusters, labels))


def test_label_time_of_many_clusters(engine):
    """Labels of a tree of 60 times as many clusters take no 15 times as long
    (by one block whatever their number, 41 times)."""
    import torch

    from fast_hdbscan_gb300 import _native

    V, lib = _native.vptr, _native.load()

    def label_ms(C):
        g = torch.Generator(device="cuda").manual_seed(C)
        n, i64 = 10 * C, torch.int64
        up = torch.rand(C - 1, generator=g, device="cuda") * torch.arange(1, C, device="cuda")
        up = up.to(i64)
        parent = torch.cat([n + up, n + torch.arange(C, device="cuda").repeat_interleave(10)])
        child = torch.cat([n + torch.arange(1, C, device="cuda"), torch.arange(n, device="cuda")])
        lam = torch.rand(n + C - 1, generator=g, device="cuda")
        size = torch.cat([torch.full((C - 1,), 10.0, device="cuda"), torch.ones(n, device="cuda")])
        sel = torch.arange(n + 1, n + C, 2, device="cuda")
        labels = torch.empty(n, dtype=i64, device="cuda")
        probs = torch.empty(n, device="cuda")
        times = []
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            _native.check(lib.fhg_label_points(
                V(parent), V(child), V(lam), V(size), parent.numel(), V(sel), sel.numel(), 0.0, n,
                V(labels), V(probs), _native.stream_ptr()))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert label_ms(1_000_000) < 15 * label_ms(16_384)


@pytest.mark.parametrize("m", [2047, 2048, 2049, 5000, 300_000])
@pytest.mark.parametrize("run", [1, 2, 9, 10, 255, 256, 257, 513, "mixed", "all"])
def test_mst_sort_runs_of_equal_weights(engine, m, run):
    """Runs of equal weight on both sides of those ordered by counting, alone
    and side by side, with repeated ends (order of arrival decides)."""
    from fast_hdbscan_gb300.cluster_trees import sort_mst

    rng = np.random.default_rng(m)
    if run == "mixed":
        lens = rng.choice([1, 1, 1, 2, 3, 40, 255, 256, 257, 1000], size=m)
        w = np.repeat(np.arange(m), lens)[:m].astype(np.float64)
    else:
        w = np.floor(np.arange(m) / (m if run == "all" else run))
    child = np.arange(1, m + 1)
    parent = np.minimum((rng.random(m) * child).astype(np.int64), rng.integers(0, 50, size=m))
    mst = np.stack([parent, child, w], axis=1).astype(np.float64)[rng.permutation(m)]
    expect = mst[np.lexsort((mst[:, 1], mst[:, 0], mst[:, 2]))]
    np.testing.assert_array_equal(sort_mst(mst), expect)


@pytest.mark.parametrize("m,most", [(2000, 1.5), (1_000_000, 0.95)])
def test_mst_sort_time_of_equal_weights(engine, m, most):
    """Sorting and linking edges of one weight against distinct weights (2.35
    and 1.08 times as long, where every edge walked its run)."""
    import torch

    from fast_hdbscan_gb300 import _native

    V, lib = _native.vptr, _native.load()

    def sort_ms(equal):
        g = torch.Generator(device="cuda").manual_seed(m)
        child = torch.arange(1, m + 1, device="cuda", dtype=torch.float64)
        u = torch.rand(2, m, generator=g, device="cuda", dtype=torch.float64)
        w = torch.full_like(child, 0.5) if equal else u[1]
        mst = torch.stack([torch.floor(u[0] * child), child, w], 1)
        mst = mst[torch.randperm(m, generator=g, device="cuda")].contiguous()
        out = torch.empty_like(mst)
        times = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            _native.check(lib.fhg_sort_mst(V(mst), m, V(out), _native.stream_ptr()))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert sort_ms(True) < most * sort_ms(False)


@pytest.mark.parametrize("m", [100, 5000, 100_000])
@pytest.mark.parametrize("weights", ["random", "few"])
def test_sort_mst_in_a_graph(engine, m, weights):
    """fhg_sort_mst asks the host for nothing, so that a CUDA graph can hold it:
    captured on one input, replayed on another."""
    import torch

    from fast_hdbscan_gb300 import _native

    rng = np.random.default_rng(m)

    def tree():
        child = np.arange(1, m + 1)
        w = rng.integers(0, 5, size=m) if weights == "few" else rng.normal(size=m) ** 2
        return np.stack([(rng.random(m) * child).astype(np.int64), child, w],
                        axis=1).astype(np.float64)

    V, lib = _native.vptr, _native.load()
    first, second = tree(), tree()
    d = torch.from_numpy(first).cuda()
    out = torch.empty_like(d)
    _native.check(lib.fhg_sort_mst(V(d), m, V(out), _native.stream_ptr()))  # kernels loaded
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _native.check(lib.fhg_sort_mst(V(d), m, V(out), _native.stream_ptr()))
    for mst in (first, second):
        d.copy_(torch.from_numpy(mst))
        graph.replay()
        expect = mst[np.lexsort((mst[:, 1], mst[:, 0], mst[:, 2]))]
        np.testing.assert_array_equal(out.cpu().numpy(), expect)
