"""The spatial index at the edges of its chunks and levels: the kNN over it
equals the oracle's whatever order the points are laid out in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 1023, 1024, 1025, 2047, 2048, 2049, 3000, 4097,
                               33_000])
@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 6, 8, 9, 17])
@pytest.mark.parametrize("kind", ["normal", "grid"])
def test_knn_over_layout_vs_oracle(engine, n, d, kind):
    from fast_hdbscan_gb300.numba_kdtree import build_kdtree, parallel_tree_query
    from oracle import oracle as O

    if n == 33_000 and (kind == "grid" or d > 5):
        pytest.skip("covered by the smaller sizes")
    rng = np.random.default_rng(100 * n + d)
    if kind == "grid":  # equal coordinates on both sides of every median
        X = rng.integers(-2, 3, size=(n, d)).astype(np.float32)
    else:
        X = (rng.normal(size=(n, d)) * np.exp(rng.normal(size=(n, 1)))).astype(np.float32)
    k = 5
    tree = build_kdtree(X)
    rd, ix = parallel_tree_query(tree, tree.data, k=k, output_rdist=True)
    ord_, oix = O.tree_query(O.build_kdtree(X), k, mode=1)
    np.testing.assert_array_equal(rd, ord_)
    np.testing.assert_array_equal(ix, oix)


@pytest.mark.parametrize("n", [5, 31, 95, 1000, 20_001, 97_281, 120_000])
@pytest.mark.parametrize("k", [1, 2, 8, 9, 16, 17, 24, 25, 32, 33, 64])
@pytest.mark.parametrize("kind", ["normal", "grid"])
def test_knn_list_lengths_vs_oracle(engine, n, k, kind):
    """Every list length's kernel, with several warps per bucket and with one,
    and with many points at the k-th distance (grid)."""
    from fast_hdbscan_gb300.numba_kdtree import build_kdtree, parallel_tree_query
    from oracle import oracle as O

    if n > 90_000 and (kind == "grid" or k not in (2, 16, 33)):
        pytest.skip("covered by the smaller sizes")
    rng = np.random.default_rng(n + 7 * k)
    d = 2 + k % 3
    if kind == "grid":
        X = rng.integers(0, 9, size=(n, d)).astype(np.float32)
    else:
        X = (rng.normal(size=(n, d)) * np.exp(rng.normal(size=(n, 1)))).astype(np.float32)
    tree = build_kdtree(X)
    rd, ix = parallel_tree_query(tree, tree.data, k=k, output_rdist=True)
    ord_, oix = O.tree_query(O.build_kdtree(X), k, mode=1)
    np.testing.assert_array_equal(rd, ord_)
    np.testing.assert_array_equal(ix, oix)


@pytest.mark.parametrize("n", [5, 600, 1025, 2600, 40_001])
@pytest.mark.parametrize("k,d", [(65, 3), (112, 2), (128, 4), (129, 1), (700, 3), (1150, 2),
                                 (2048, 3), (101, 11), (90, 20)])
@pytest.mark.parametrize("kind", ["normal", "grid", "same"])
def test_long_knn_lists_vs_oracle(engine, n, k, d, kind):
    """Lists longer than 64, from fewer points than k to trees of several
    levels of 32, with many points at the k-th distance (grid) and, in the
    buffer's cuts, keys that differ in their index alone (same)."""
    from fast_hdbscan_gb300.numba_kdtree import build_kdtree, parallel_tree_query
    from oracle import oracle as O

    if n > 3000 and (kind == "same" or d > 4 or k > 1200):
        pytest.skip("covered by the smaller sizes")
    rng = np.random.default_rng(n + 7 * k + d)
    if kind == "normal":
        X = (rng.normal(size=(n, d)) * np.exp(rng.normal(size=(n, 1)))).astype(np.float32)
    else:
        X = rng.integers(0, 9 if kind == "grid" else 2, size=(n, d)).astype(np.float32)
    tree = build_kdtree(X)
    rd, ix = parallel_tree_query(tree, tree.data, k=k, output_rdist=True)
    ord_, oix = O.tree_query(O.build_kdtree(X), k, mode=1)
    np.testing.assert_array_equal(rd, ord_)
    np.testing.assert_array_equal(ix, oix)


@pytest.mark.parametrize("m", [2, 2048, 2049, 2816, 2817, 4096, 4097, 8192, 8193, 100_001,
                               1_000_000])
@pytest.mark.parametrize("weights", ["random", "few", "equal"])
def test_mst_sort_sizes(engine, m, weights):
    """The radix sort at the edges of its tiles, through the MST sort (float64
    weights: keys of 64 and 32 bits), against np.lexsort."""
    from fast_hdbscan_gb300.cluster_trees import sort_mst

    rng = np.random.default_rng(m)
    w = {"random": rng.normal(size=m) ** 2, "few": rng.integers(0, 5, size=m) / 4.0,
         "equal": np.full(m, 0.5)}[weights]
    # a spanning tree: every point past the first hangs from an earlier one
    child = np.arange(1, m + 1)
    mst = np.stack([(rng.random(m) * child).astype(np.int64), child, w], axis=1).astype(np.float64)
    mst = mst[rng.permutation(m)]
    expect = mst[np.lexsort((mst[:, 1], mst[:, 0], mst[:, 2]))]
    np.testing.assert_array_equal(sort_mst(mst), expect)


@pytest.mark.parametrize("mcs", [1, 2, 31, 511, 512, 513, 2500])
@pytest.mark.parametrize("n", [7000, 20_000])
def test_condense_segments_vs_oracle(engine, n, mcs):
    """Condensed rows ordered by counting (short segments) and by sorting."""
    from fast_hdbscan_gb300 import synthetic
    from fast_hdbscan_gb300.cluster_trees import condense_tree, mst_to_linkage_tree, sort_mst
    from oracle import oracle as O

    X = synthetic.varying_density(n, seed=mcs)
    mst = O.parallel_boruvka(O.build_kdtree(X), 5, mode=1)[0]
    linkage = mst_to_linkage_tree(sort_mst(mst))
    got, expect = condense_tree(linkage, min_cluster_size=mcs), O.condense_tree(linkage, mcs)
    for a, b in zip(got, expect):
        np.testing.assert_array_equal(a, b)


def _far_groups(n, d, far, seed):
    """n points, `far` of them 1e20 from the rest: finite rows whose squared
    distances overflow float32."""
    X = np.random.default_rng(seed).normal(size=(n, d)).astype(np.float32)
    X[-far:, 0] += np.float32(1e20)
    return X[np.random.default_rng(seed + 1).permutation(n)]


@pytest.mark.parametrize("n,far", [(65, 3), (90, 5), (129, 64), (1000, 7), (2049, 20),
                                   (4097, 2000), (5000, 9)])
@pytest.mark.parametrize("d", [1, 3, 5, 7, 20])
@pytest.mark.parametrize("k", [2, 11, 24, 40])
def test_knn_at_infinite_distances_vs_oracle(engine, n, far, d, k):
    """Lists that must be filled with points at infinite distances, where the
    tree has slots without points: by index, each point once."""
    from fast_hdbscan_gb300.numba_kdtree import build_kdtree, parallel_tree_query
    from oracle import oracle as O

    X = _far_groups(n, d, far, 10 * n + d)
    tree = build_kdtree(X)
    rd, ix = parallel_tree_query(tree, tree.data, k=k, output_rdist=True)
    ord_, oix = O.tree_query(O.build_kdtree(X), k, mode=1)
    np.testing.assert_array_equal(rd, ord_)
    np.testing.assert_array_equal(ix, oix)


def test_knn_does_not_scan_empty_slots(engine):
    """One point in the last bucket, beside as many slots without points as the
    tree can have: the walk that fills its list costs no more than others."""
    import ctypes

    import torch

    from fast_hdbscan_gb300 import _native

    V, lib, k = _native.vptr, _native.load(), 16

    def knn_ms(n):
        g = torch.Generator(device="cuda").manual_seed(3)
        X = torch.randn(n, 3, generator=g, device="cuda")
        rd = torch.empty(n, k, device="cuda")
        ix = torch.empty(n, k, dtype=torch.int32, device="cuda")
        h = ctypes.c_void_p()
        _native.check(lib.fhg_index_build(V(X), n, 3, _native.stream_ptr(), ctypes.byref(h)))
        times = []
        for _ in range(4):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            _native.check(lib.fhg_index_knn(h, k, V(rd), V(ix), _native.stream_ptr()))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        _native.check(lib.fhg_index_free(h, _native.stream_ptr()))
        return min(times)

    assert knn_ms(2**20 + 1) < 3 * knn_ms(2**20)


@pytest.mark.parametrize("n", [70, 3000, 50_000])
@pytest.mark.parametrize("copies", [20, 200])
@pytest.mark.parametrize("order", ["together", "mixed"])
@pytest.mark.parametrize("k", [2, 8, 11, 16, 24, 31, 40, 64])
def test_knn_among_equal_points_vs_oracle(engine, n, copies, order, k):
    """Buckets of nothing but equal points: more candidates at once than a
    query's queue has room for, before and after its list."""
    from fast_hdbscan_gb300.numba_kdtree import build_kdtree, parallel_tree_query
    from oracle import oracle as O

    rng = np.random.default_rng(n + copies + k)
    d = 2 + k % 5
    X = np.repeat(rng.normal(size=(n // copies + 1, d)), copies, axis=0)[:n].astype(np.float32)
    if order == "mixed":
        X = X[rng.permutation(n)]
    tree = build_kdtree(X)
    rd, ix = parallel_tree_query(tree, tree.data, k=k, output_rdist=True)
    ord_, oix = O.tree_query(O.build_kdtree(X), k, mode=1)
    np.testing.assert_array_equal(rd, ord_)
    np.testing.assert_array_equal(ix, oix)


def test_knn_time_among_equal_points(engine):
    """Equal points cost what their distances cost, not a merge for every eight
    that could join no list (7.5 times the kNN of distinct points before)."""
    import torch

    from fast_hdbscan_gb300 import _native

    V, lib, k, n = _native.vptr, _native.load(), 16, 300_000

    def knn_ms(X):
        import ctypes

        rd = torch.empty(n, k, device="cuda")
        ix = torch.empty(n, k, dtype=torch.int32, device="cuda")
        h = ctypes.c_void_p()
        _native.check(lib.fhg_index_build(V(X), n, 3, _native.stream_ptr(), ctypes.byref(h)))
        times = []
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            _native.check(lib.fhg_index_knn(h, k, V(rd), V(ix), _native.stream_ptr()))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        _native.check(lib.fhg_index_free(h, _native.stream_ptr()))
        return min(times)

    g = torch.Generator(device="cuda").manual_seed(3)
    X = torch.randn(n, 3, generator=g, device="cuda")
    assert knn_ms(X[:300].repeat_interleave(1000, 0).contiguous()) < 4.5 * knn_ms(X)
