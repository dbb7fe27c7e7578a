"""The high-dimensional route (hdbscan.py:446 -> nndescent.py:179
compute_mst_from_knn_graph) on the GPU's exact brute-force kNN.

* The tensor-core kNN with its certified float32 re-rank equals the spatial
  index's kNN bit for bit where both exist (d <= 32) and the CPU oracle's
  exact kNN at 64 dimensions, including inputs whose certificate fails
  (duplicated points) and go through the exact fallback.
* Core distances agree with a float64 brute force within 1e-5 relative.
* The kNN-graph forest and the whole fit equal the oracle's Kruskal on the
  oracle's exact kNN lists (pynndescent's graph is approximate; the exact
  graph is what it converges to).
"""
import ctypes
import os

import numpy as np
import pytest

from fast_hdbscan_gb300 import synthetic

pytestmark = pytest.mark.gpu
NTH = os.cpu_count() or 1


def _highd(X, k):
    import torch

    from fast_hdbscan_gb300 import _native

    Xd = torch.from_numpy(np.ascontiguousarray(X, np.float32)).cuda()
    n, d = X.shape
    rd = torch.empty((n, k), dtype=torch.float32, device="cuda")
    ix = torch.empty((n, k), dtype=torch.int32, device="cuda")
    fb = ctypes.c_int64(0)
    _native.check(_native.load().fhg_highd_knn(_native.vptr(Xd), n, d, k, _native.vptr(rd),
                                               _native.vptr(ix), ctypes.byref(fb),
                                               _native.stream_ptr()))
    return rd.cpu().numpy(), ix.cpu().numpy(), fb.value


@pytest.mark.parametrize("d,k", [(12, 11), (24, 31), (32, 16), (3, 5)])
def test_highd_knn_equals_spatial_knn(engine, d, k):
    from fast_hdbscan_gb300.numba_kdtree import build_kdtree, parallel_tree_query

    X = synthetic.aniso_highdim(n=6000, seed=20 + d, dim=d, n_comp=8)
    rd, ix, fb = _highd(X, k)
    rd_t, ix_t = parallel_tree_query(build_kdtree(X), X, k=k, output_rdist=True)
    np.testing.assert_array_equal(ix, ix_t)
    np.testing.assert_array_equal(rd, rd_t)


@pytest.mark.parametrize("d", [40, 64, 96])
def test_highd_knn_equals_oracle(engine, d):
    from oracle import oracle as O

    X = synthetic.aniso_highdim(n=8000, seed=30 + d, dim=d, n_comp=10)
    k = 31
    rd, ix, fb = _highd(X, k)
    rd_o, ix_o = O.tree_query(O.build_kdtree(X), k, mode=1, nthreads=NTH)
    np.testing.assert_array_equal(ix, ix_o)
    np.testing.assert_array_equal(rd, rd_o)
    print("d=%d fallbacks %d of %d" % (d, fb, len(X)))
    # float64 brute force on a sample of queries: the k-th distance
    rows = np.random.default_rng(d).choice(len(X), 64, replace=False)
    X64 = X.astype(np.float64)
    for i in rows:
        dd = np.sort(((X64 - X64[i]) ** 2).sum(1))
        assert abs(np.sqrt(rd[i, -1]) - np.sqrt(dd[k - 1])) <= 1e-5 * np.sqrt(dd[k - 1])


def test_highd_knn_fallback_path(engine):
    """Many copies of a few points: the L-th candidate estimate is 0, no
    certificate holds, and the exact fallback answers every such query."""
    from oracle import oracle as O

    rng = np.random.default_rng(7)
    base = rng.normal(0, 1, (20, 48)).astype(np.float32)
    X = np.concatenate([np.repeat(base, 60, axis=0),
                        rng.normal(0, 3, (800, 48)).astype(np.float32)])
    X = X[rng.permutation(len(X))]
    rd, ix, fb = _highd(X, 16)
    assert fb >= 1200
    rd_o, ix_o = O.tree_query(O.build_kdtree(X), 16, mode=1, nthreads=NTH)
    np.testing.assert_array_equal(ix, ix_o)
    np.testing.assert_array_equal(rd, rd_o)


@pytest.mark.parametrize("ms,knn_k", [(10, None), (5, 20), (1, None)])
def test_knn_graph_mst_equals_oracle(engine, ms, knn_k):
    from fast_hdbscan_gb300.hdbscan import compute_minimum_spanning_tree, resolve_knn_graph_k
    from oracle import oracle as O

    X = synthetic.aniso_highdim(n=5000, seed=41, dim=64, n_comp=6)
    mst, nbrs, core = compute_minimum_spanning_tree(X, min_samples=ms, knn_k=knn_k)
    kk = resolve_knn_graph_k(ms, knn_k)
    e_o, n_o, c_o = O.kruskal_knn(O.build_kdtree(X), ms, kk, mode=1, nthreads=NTH)
    np.testing.assert_array_equal(mst, e_o)
    np.testing.assert_array_equal(nbrs, n_o)
    np.testing.assert_array_equal(core, c_o)


def test_knn_graph_fit_equals_oracle(engine):
    from fast_hdbscan_gb300 import HDBSCAN
    from fast_hdbscan_gb300.hdbscan import resolve_knn_graph_k
    from oracle import oracle as O

    X = synthetic.aniso_highdim(n=12000, seed=42, dim=64, n_comp=12)
    est = HDBSCAN(min_samples=10, min_cluster_size=100).fit(X)
    mst, _, _ = O.kruskal_knn(O.build_kdtree(X), 10, resolve_knn_graph_k(10, None), mode=1,
                              nthreads=NTH)
    labels, probs, *_ = O.clusters_from_spanning_tree(mst, min_cluster_size=100)
    np.testing.assert_array_equal(est.labels_, labels)
    np.testing.assert_array_equal(est.probabilities_, probs)
    assert len(set(labels.tolist()) - {-1}) >= 2


@pytest.mark.parametrize("n,d,k", [(100, 40, 5), (1000, 20, 31), (4999, 64, 31),
                                   (20_000, 64, 16), (40_000, 48, 31), (3000, 64, 32),
                                   (3000, 64, 36)])
def test_tcgen05_pipeline_equals_mma_sync_kernel(engine, n, d, k):
    """The tcgen05 candidate pipeline (TMA, tensor memory, epilogue
    selection) and the mma.sync kernel give the same certified kNN, equal to
    the oracle's exact kNN -- on ragged last tiles, on fewer points than
    one tile, and on both sides of the largest candidate buffers the
    pipeline's shared memory holds (k 32 runs on tcgen05, k 36 falls back)."""
    from fast_hdbscan_gb300 import _native
    from oracle import oracle as O

    X = synthetic.aniso_highdim(n=n, seed=50 + d, dim=d, n_comp=7)
    lib = _native.load()
    assert lib.fhg_set_highd_kernel(0) == 0
    rd_tc, ix_tc, fb_tc = _highd(X, k)
    lib.fhg_set_highd_kernel(1)
    try:
        rd_ms, ix_ms, fb_ms = _highd(X, k)
    finally:
        lib.fhg_set_highd_kernel(0)
    np.testing.assert_array_equal(ix_tc, ix_ms)
    np.testing.assert_array_equal(rd_tc, rd_ms)
    rd_o, ix_o = O.tree_query(O.build_kdtree(X), k, mode=1, nthreads=NTH)
    np.testing.assert_array_equal(ix_tc, ix_o)
    np.testing.assert_array_equal(rd_tc, rd_o)
    print("n=%d d=%d k=%d: fallbacks tcgen05 %d, mma.sync %d" % (n, d, k, fb_tc, fb_ms))


@pytest.mark.parametrize("n,d,k", [(127, 33, 31), (128, 64, 31), (129, 32, 31), (3969, 31, 4),
                                   (4096, 64, 1), (4097, 63, 31), (6000, 33, 31), (6001, 32, 56),
                                   (6000, 32, 57), (4200, 30, 56), (4100, 64, 48),
                                   (4100, 64, 49)])
def test_tcgen05_tiles_and_thresholds_equal_oracle(engine, n, d, k):
    """Around a tile of 128, around the 32 tiles from which first thresholds
    are taken, dimensions that fill their segment or leave one over (with and
    without 16-byte rows), and the lists around the largest buffers: the
    oracle's lists exactly.  A tight group far from the rest, and a row of
    duplicates, want candidates that first thresholds must not cut off."""
    from oracle import oracle as O

    X = synthetic.aniso_highdim(n=n, seed=70 + d, dim=d, n_comp=5)
    X[: n // 20] = X[0] * 3 + 0.01 * X[: n // 20]
    X[n // 2: n // 2 + min(k, 40)] = X[n // 2]
    rd, ix, _ = _highd(X, k)
    rd_o, ix_o = O.tree_query(O.build_kdtree(X), k, mode=1, nthreads=NTH)
    np.testing.assert_array_equal(ix, ix_o)
    np.testing.assert_array_equal(rd, rd_o)


@pytest.mark.parametrize("n,d,k", [(1000, 40, 5), (4201, 33, 31), (4097, 64, 16)])
def test_rows_near_the_largest_float_equal_brute_force(engine, n, d, k):
    """Finite rows whose bfloat16 parts are infinite give estimates that are no
    numbers, in the columns past the last point too: these are no candidates."""
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, d)).astype(np.float32)
    big = np.finfo(np.float32).max
    X[[3, n // 3, n // 2, n - 1]] = np.array([[big], [-big], [big], [-big]], np.float32)
    rd, ix, _ = _highd(X, k)
    with np.errstate(over="ignore"):
        for i in np.concatenate([[3, n // 3, n // 2, n - 1], rng.choice(n, 60, replace=False)]):
            dd = np.zeros(n, np.float32)
            for j in range(d):
                dd += (X[i, j] - X[:, j]) ** 2
            order = np.lexsort((np.arange(n), dd))[:k]
            np.testing.assert_array_equal(ix[i], order)
            np.testing.assert_array_equal(rd[i], dd[order])


@pytest.mark.parametrize("n,d,k", [(4096, 64, 1), (4097, 63, 31), (6001, 32, 56), (4100, 64, 48)])
def test_first_thresholds_leave_rows_certified(engine, n, d, k):
    """A first threshold that cut off candidates would show in the rows that
    are searched again, not in the lists.  Both kernels certify a row by its
    L-th smallest estimate, computed from the same products: only rows within
    rounding of the bound may differ, 1 % of them at most."""
    from fast_hdbscan_gb300 import _native

    X = synthetic.aniso_highdim(n=n, seed=70 + d, dim=d, n_comp=5)
    X[: n // 20] = X[0] * 3 + 0.01 * X[: n // 20]
    lib = _native.load()
    _, _, fb_tc = _highd(X, k)
    lib.fhg_set_highd_kernel(1)
    try:
        _, _, fb_ms = _highd(X, k)
    finally:
        lib.fhg_set_highd_kernel(0)
    print("n=%d d=%d k=%d: fallbacks tcgen05 %d, mma.sync %d" % (n, d, k, fb_tc, fb_ms))
    assert fb_tc <= fb_ms + n // 100


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("scale", [1e19, 1e20, 1e38])
@pytest.mark.parametrize("n,d,k", [(90, 33, 16), (1000, 40, 11), (4500, 64, 31), (3000, 70, 5)])
def test_overflowing_estimates_equal_brute_force(engine, kernel, scale, n, d, k):
    """Groups of finite rows so far apart that |y|^2 overflows: no estimate says
    anything, so no row may be certified by them."""
    from fast_hdbscan_gb300 import _native

    rng = np.random.default_rng(n + d)
    X = rng.normal(size=(n, d))
    X[:, 3] += scale * rng.integers(0, 3, n)
    X = X.astype(np.float32)
    lib = _native.load()
    lib.fhg_set_highd_kernel(kernel)
    try:
        rd, ix, _ = _highd(X, k)
    finally:
        lib.fhg_set_highd_kernel(0)
    with np.errstate(over="ignore"):
        for i in rng.choice(n, 60, replace=False):
            dd = np.zeros(n, np.float32)
            for j in range(d):
                dd += (X[i, j] - X[:, j]) ** 2
            order = np.lexsort((np.arange(n), dd))[:k]
            np.testing.assert_array_equal(ix[i], order)
            np.testing.assert_array_equal(rd[i], dd[order])
