// kNN-graph Kruskal MST (kruskal.py:950 _kruskal_mst_knn, the
// algorithm="kruskal" back-end with an integer knn_k, without cannot-link
// constraints).
//
// The reference lists the mutual-reachability edges of every point's kNN list
// (kruskal.py:456), drops self-loops and infinite weights, orders them by a
// stable argsort of their float64 weights and runs Kruskal's union-find; a
// disconnected kNN graph is then joined by +inf bridges between the smallest
// points of its components (kruskal.py:723, precomputed.py:308).
//
// Here: the spatial index's kNN (rows in caller order), one thread per edge
// for the weights, a stable LSD radix sort of the valid edges, and -- in place
// of the sequential scan -- Boruvka rounds over the sorted ranks: every
// component takes its lowest-rank outgoing edge, the picked edges are hooked
// with a lock-free union-find and edges inside one component leave the active
// list.  Ranks are distinct, so the forest is the one Kruskal accepts (the
// minimum spanning forest of a strict order is unique); compacting the picked
// ranks gives Kruskal's acceptance order.  The union-find keeps every root the
// smallest point of its component, so the bridges join the roots in index
// order.
//
// Every float64 weight is a monotone image of one float32 value -- without
// sample weights sqrt(double(max(core2_i, core2_j, rdist_ij))) (core2 the
// squared core distance, a kNN rdist entry), with them
// double(max(core_i, core_j, sqrtf(rdist_ij))) -- and distinct float32 values
// give distinct weights (a correctly rounded double square root keeps the
// strict order of float32 inputs), so the sort runs on the 32-bit pattern of
// that value (non-negative floats order like their bits).
#include <memory>

#include "compact.cuh"
#include "highd.cuh"
#include "index.cuh"
#include "mst.cuh"
#include "primitives.cuh"
#include "uf.cuh"

namespace fhg {
namespace {

#define LAUNCH(kernel, count, ...)                                        \
    do {                                                                  \
        if ((count) > 0) {                                                \
            ::fhg::note_launch();                                         \
            kernel<<<grid_for((count), 256), 256, 0, s>>>(__VA_ARGS__);   \
            FHG_CUDA(cudaGetLastError());                                 \
        }                                                                 \
    } while (0)

// kruskal.py:995-1015: float64 core distances from the kNN lists (rows of kq,
// the point itself first; min_samples <= 1: zero) and the float32 value the
// edge keys take the maximum of (the squared core distance), beside the squared
// distance of the point's last neighbour (+inf when the row is not full).
__device__ __forceinline__ float kr_last(int64_t i, int kq, const float* __restrict__ rd,
                                         const int32_t* __restrict__ ix) {
    return ix[i * kq + kq - 1] >= 0 ? rd[i * kq + kq - 1] : INFINITY;
}
__global__ void kr_core_kernel(int64_t n, int kq, int ms, const float* __restrict__ rd,
                               const int32_t* __restrict__ ix, double* __restrict__ core,
                               float2* __restrict__ ck) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float c2 = ms > 1 ? rd[i * kq + ms] : 0.0f;
    core[i] = ms > 1 ? __dsqrt_rn((double)c2) : 0.0;
    ck[i] = make_float2(c2, kr_last(i, kq, rd, ix));
}
// kruskal.py:981-990 with boruvka.py:528 sample_weight_core_distance: the
// first list position at which the running float64 weight (the point's own
// first) reaches min_samples; index -1 (padding) reads the last weight.  The
// distances are the float32 square roots the reference's tree query returns.
__global__ void kr_core_w_kernel(int64_t n, int kq, int ms, const float* __restrict__ rd,
                                 const int32_t* __restrict__ ix, const float* __restrict__ w,
                                 double* __restrict__ core, float2* __restrict__ ck) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double total = 0.0;
    int j = 0;
    while (total < (double)ms && j < kq) {
        const int32_t q = ix[i * kq + j];
        total += (double)w[q >= 0 ? q : n - 1];
        ++j;
    }
    const float c = __fsqrt_rn(rd[i * kq + (j > 0 ? j - 1 : 0)]);
    core[i] = (double)c;
    ck[i] = make_float2(c, kr_last(i, kq, rd, ix));
}
// kruskal.py:456 _build_mrd_edges_knn and the filter of :1022, as each edge's
// float32 key (kNoEdge: filtered out).  Edge e is the (e % kk)-th neighbour of
// point e / kk (kk = kq - 1).  An edge from i to a smaller j that lies within
// j's last distance stands in j's row too: with the same weight and, the rows
// being in order, an earlier place, so the later one is never accepted and is
// left out here (3-D, 16 neighbours: two thirds of the edges are left to sort).
constexpr uint32_t kNoEdge = 0xffffffffu;  // (a NaN: no key of a finite weight)
__global__ void kr_edges_kernel(int64_t n, int kq, int weighted, const float* __restrict__ rd,
                                const int32_t* __restrict__ ix, const float2* __restrict__ ck,
                                uint32_t* __restrict__ key) {
    const uint32_t kk = (uint32_t)(kq - 1);
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * kk) return;  // (at most 2^31 - 1 edges)
    const int64_t i = (uint32_t)e / kk, at = i * kq + (e - i * kk) + 1;
    const int32_t j = ix[at];
    uint32_t out = kNoEdge;
    if (j >= 0 && j != (int32_t)i) {
        const float r = rd[at];
        const float2 cj = ck[j];
        const float v = fmaxf(fmaxf(ck[i].x, cj.x), weighted ? __fsqrt_rn(r) : r);
        if (isfinite(v) && !(j < (int32_t)i && r < cj.y)) out = __float_as_uint(v);
    }
    key[e] = out;
}
// The edges that are left, in order.
struct KeptEdges {
    const uint32_t* k0;
    uint32_t* key;
    int32_t* eid;
    __device__ bool test(int64_t e) const { return k0[e] != kNoEdge; }
    __device__ void emit(int64_t e, uint32_t at) const {
        key[at] = k0[e];
        eid[at] = (int32_t)e;
    }
    __device__ void each(int64_t) const {}
};
// Endpoints of every sorted edge.
__global__ void kr_ends_kernel(int64_t m, int kq, const int32_t* __restrict__ eid,
                               const int32_t* __restrict__ ix, int2* __restrict__ uv) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    const uint32_t kk = (uint32_t)(kq - 1), e = (uint32_t)eid[r], i = e / kk;
    uv[r] = make_int2((int32_t)i, ix[(int64_t)i * kq + (e - i * kk) + 1]);
}
__global__ void kr_init_kernel(int64_t n, int32_t* __restrict__ par, uint32_t* __restrict__ best) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    par[i] = (int32_t)i;
    best[i] = 0xffffffffu;
}
// One Boruvka round over the active edges (rank act[t], or t in the first
// round; act_uv their components).  What bounds it is the gathers by component:
// endpoints are looked up once a round, by the compaction that ends it, the
// picked edges are joined by a pass over the points, and a round takes five
// launches (16M edges of 1M points: 2.2 -> 0.8 ms; 4.5M pairs of 300k points,
// twice as many entries before: 1.5 -> 0.5).
// Step 1: every component's lowest outgoing rank.  Active ranks come in
// increasing order, so a component's best is mostly set by its first edge and
// later ones only read it.
__global__ void kr_best_kernel(int64_t na, const int32_t* __restrict__ act,
                               const int2* __restrict__ act_uv, uint32_t* __restrict__ best) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= na) return;
    const uint32_t r = act ? (uint32_t)act[t] : (uint32_t)t;
    const int2 p = act_uv[t];
    if (p.x == p.y) return;
    if (r < *(volatile uint32_t*)&best[p.x]) atomicMin(&best[p.x], r);
    if (r < *(volatile uint32_t*)&best[p.y]) atomicMin(&best[p.y], r);
}
// Step 2: the picked edges are marked and hooked (an edge that both of its
// components pick, twice: the second union finds nothing to do).
__global__ void kr_join_kernel(int64_t n, uint32_t* __restrict__ best,
                               const int2* __restrict__ uv, uint8_t* __restrict__ mark,
                               int32_t* par) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const uint32_t r = best[c];
    if (r == 0xffffffffu) return;
    best[c] = 0xffffffffu;
    mark[r] = 1;
    const int2 p = uv[r];
    uf_union(par, p.x, p.y);
}
// Step 3: every point's parent is its root.  (Reads the chains only: a find that
// halves paths could put an inner point back behind another thread's root.)
__global__ void kr_flatten_kernel(int64_t n, int32_t* par) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t first = par[i];
    int32_t root = first, up;
    while ((up = par[root]) != root) root = up;
    if (root != first) par[i] = root;
}
// Step 4: edges between two components stay.
struct EdgesApart {
    const int32_t* act;
    const int2* act_uv;
    const int32_t* par;
    int32_t* act2;
    int2* act_uv2;
    __device__ bool test(int64_t t) const {
        const int2 p = act_uv[t];
        return par[p.x] != par[p.y];
    }
    __device__ void emit(int64_t t, uint32_t at) const {
        const int2 p = act_uv[t];
        act2[at] = act ? act[t] : (int32_t)t;
        act_uv2[at] = make_int2(par[p.x], par[p.y]);
    }
    __device__ void each(int64_t) const {}
};
// The picked ranks in order, and kruskal.py:104-107: their edges as (row point,
// neighbour, float64 weight); the weight is the rank's float32 key (kNN graph)
// or its float64 weight.  (The float64 square roots want full warps: taken in
// the compaction, a few lanes at a time, they made it 250 us at 1M points.)
struct PickedRanks {
    const uint8_t* mark;
    int32_t* ranks;
    __device__ bool test(int64_t r) const { return mark[r] != 0; }
    __device__ void emit(int64_t r, uint32_t at) const { ranks[at] = (int32_t)r; }
    __device__ void each(int64_t) const {}
};
__global__ void kr_emit_kernel(int64_t nf, int weighted, const int32_t* __restrict__ ranks,
                               const int2* __restrict__ uv, const uint32_t* __restrict__ key,
                               const double* __restrict__ w64, double* __restrict__ edges) {
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= nf) return;
    const int32_t r = ranks[o];
    const int2 p = uv[r];
    edges[3 * o + 0] = (double)p.x;
    edges[3 * o + 1] = (double)p.y;
    if (w64) {
        edges[3 * o + 2] = w64[r];
    } else {
        const float v = __uint_as_float(key[r]);
        edges[3 * o + 2] = weighted ? (double)v : __dsqrt_rn((double)v);
    }
}
struct ForestRoots {
    const int32_t* par;
    int32_t* roots;
    __device__ bool test(int64_t i) const { return par[i] == (int32_t)i; }
    __device__ void emit(int64_t i, uint32_t at) const { roots[at] = (int32_t)i; }
    __device__ void each(int64_t) const {}
};
// kruskal.py:723 / precomputed.py:308: +inf bridges between consecutive
// component representatives (the roots, each its component's smallest point).
__global__ void kr_bridge_kernel(int64_t nb, const int32_t* __restrict__ roots,
                                 double* __restrict__ edges) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nb) return;
    edges[3 * c + 0] = (double)roots[c];
    edges[3 * c + 1] = (double)roots[c + 1];
    edges[3 * c + 2] = INFINITY;
}
__global__ void kr_neighbors_kernel(int64_t n, int kq, int cols, const int32_t* __restrict__ ix,
                                    int32_t* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * cols) return;
    const int64_t i = t / cols, c = t - i * cols;
    out[t] = ix[i * kq + c + 1];
}

}  // namespace

int kruskal_knn_mst(const fhg_index& index, int min_samples, int query_k, const float* weights,
                    double* edges, int32_t* neighbors, double* core, int64_t* n_components,
                    cudaStream_t s) {
    return kruskal_mst_of_lists(index.n, min_samples, query_k, weights, &index, nullptr, 0,
                                edges, neighbors, core, n_components, s);
}

int kruskal_mst_of_lists(int64_t n, int min_samples, int query_k, const float* weights,
                         const fhg_index* index, const float* X, int d, double* edges,
                         int32_t* neighbors, double* core, int64_t* n_components,
                         cudaStream_t s) {
    const int kq = query_k;
    const int64_t kk = kq - 1;
    // the spatial index's kNN takes lists of up to kKnnMaxK; the
    // high-dimensional kNN graph is used here with lists of up to 64
    const int kq_max = index ? kKnnMaxK : 64;
    if (kq < 2 || kq > kq_max) {
        set_error("kruskal: the kNN query size must be in [2, %d] (got %d)", kq_max, kq);
        return kq > kq_max ? FHG_ERR_UNSUPPORTED : FHG_ERR_INVALID;
    }
    if (n * kk > 0x7fffffffLL) {
        set_error("kruskal: %lld kNN edges exceed the int32 edge index", (long long)(n * kk));
        return FHG_ERR_UNSUPPORTED;
    }
    if (!weights && min_samples > 1 && min_samples >= kq) {
        set_error("kruskal: the kNN query size %d must exceed min_samples %d", kq, min_samples);
        return FHG_ERR_INVALID;
    }
    *n_components = n > 0 ? 1 : 0;
    if (n < 2) {
        if (n == 1) FHG_CUDA(cudaMemsetAsync(core, 0, sizeof(double), s));
        return FHG_OK;
    }
    Stage stage(s, "kruskal_knn");
    Workspace ws(s);
    float* rd;
    float2* ck;
    int32_t* ix;
    FHG_TRY(ws.alloc(&rd, (size_t)(n * kq)));
    FHG_TRY(ws.alloc(&ix, (size_t)(n * kq)));
    FHG_TRY(ws.alloc(&ck, (size_t)n));
    if (index) FHG_TRY(index_knn(*index, kq, nullptr, nullptr, rd, ix, s));
    else FHG_TRY(highd_knn(X, n, d, kq, rd, ix, nullptr, s));
    if (weights) LAUNCH(kr_core_w_kernel, n, n, kq, min_samples, rd, ix, weights, core, ck);
    else LAUNCH(kr_core_kernel, n, n, kq, min_samples, rd, ix, core, ck);
    if (neighbors) {
        const int cols = weights ? kq - 1 : (min_samples > 1 ? min_samples : 1);
        LAUNCH(kr_neighbors_kernel, n * cols, n, kq, cols, ix, neighbors);
    }

    // ---- valid edges, stably sorted by weight
    std::unique_ptr<Stage> sub(new Stage(s, "kruskal_edges"));
    const int64_t E = n * kk;
    uint32_t *k0, *key, *cnt;
    int32_t* eid;
    FHG_TRY(ws.alloc(&k0, (size_t)E));
    FHG_TRY(ws.alloc(&key, (size_t)E));
    FHG_TRY(ws.alloc(&eid, (size_t)E));
    FHG_TRY(ws.alloc(&cnt, 1));
    LAUNCH(kr_edges_kernel, E, n, kq, weights ? 1 : 0, rd, ix, ck, k0);
    FHG_TRY(compact(ws, KeptEdges{k0, key, eid}, E, cnt));
    uint32_t h_m = 0;
    FHG_CUDA(cudaMemcpyAsync(&h_m, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    const int64_t m = h_m;
    sub.reset(new Stage(s, "kruskal_sort"));
    if (m > 1) {
        Workspace tmp(ws);
        FHG_TRY(radix_sort_u32(tmp, key, eid, m, 0, 32));
    }

    sub.reset();
    FHG_TRY(sorted_forest_edges(ws, n, m, kq, eid, ix, nullptr, key, weights ? 1 : 0, edges,
                                n_components));
    return FHG_OK;
}

int sorted_forest_edges(Workspace& ws, int64_t n, int64_t m, int kq, const int32_t* eid,
                        const int32_t* ix, const int2* uv_in, const uint32_t* key32,
                        int key_weighted, double* edges, int64_t* n_components,
                        const double* w64) {
    cudaStream_t s = ws.stream();
    const size_t mm = (size_t)(m > 0 ? m : 1);
    // ---- minimum spanning forest: Boruvka rounds over the ranks
    std::unique_ptr<Stage> sub(new Stage(s, "kruskal_forest"));
    int32_t *par, *act = nullptr, *act_a, *act_b;
    int2 *uv_a, *uv_b;
    const int2 *uv = uv_in, *act_uv;
    uint32_t *best, *cnt;
    uint8_t* mark;
    FHG_TRY(ws.alloc(&par, (size_t)n));
    FHG_TRY(ws.alloc(&best, (size_t)n));
    FHG_TRY(ws.alloc(&act_a, mm));
    FHG_TRY(ws.alloc(&act_b, mm));
    FHG_TRY(ws.alloc(&uv_a, mm));
    FHG_TRY(ws.alloc(&uv_b, mm));
    FHG_TRY(ws.alloc(&mark, mm));
    FHG_TRY(ws.alloc(&cnt, 1));
    LAUNCH(kr_init_kernel, n, n, par, best);
    if (!uv_in) {
        int2* ends;
        FHG_TRY(ws.alloc(&ends, mm));
        LAUNCH(kr_ends_kernel, m, m, kq, eid, ix, ends);
        uv = ends;
    }
    act_uv = uv;
    if (m > 0) FHG_CUDA(cudaMemsetAsync(mark, 0, (size_t)m, s));
    uint32_t h = 0;
    int64_t na = m;
    for (int round = 1; na > 0; ++round) {
        if (round > 64) {  // each round at least halves the components
            set_error("kruskal: the spanning forest did not converge");
            return FHG_ERR_NO_CONVERGENCE;
        }
        LAUNCH(kr_best_kernel, na, na, act, act_uv, best);
        LAUNCH(kr_join_kernel, n, n, best, uv, mark, par);
        LAUNCH(kr_flatten_kernel, n, n, par);
        FHG_TRY(compact(ws, EdgesApart{act, act_uv, par, act_a, uv_a}, na, cnt));
        FHG_CUDA(cudaMemcpyAsync(&h, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        FHG_CUDA(cudaStreamSynchronize(s));
        act = act_a;
        act_uv = uv_a;
        std::swap(act_a, act_b);
        std::swap(uv_a, uv_b);
        na = (int64_t)h;
    }

    // ---- the forest in Kruskal's acceptance order, then the bridges
    sub.reset(new Stage(s, "kruskal_emit"));
    int32_t* ranks = act_a;  // (room for all m)
    FHG_TRY(compact(ws, PickedRanks{mark, ranks}, m, cnt));
    FHG_CUDA(cudaMemcpyAsync(&h, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    const int64_t nf = h, nc = n - nf;
    if (nc >= 1) LAUNCH(kr_emit_kernel, nf, nf, key_weighted, ranks, uv, key32, w64, edges);
    if (nc > 1) {
        int32_t* roots;
        FHG_TRY(ws.alloc(&roots, (size_t)n));
        FHG_TRY(compact(ws, ForestRoots{par, roots}, n, cnt));
        FHG_CUDA(cudaMemcpyAsync(&h, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        FHG_CUDA(cudaStreamSynchronize(s));
        if ((int64_t)h == nc) LAUNCH(kr_bridge_kernel, nc - 1, nc - 1, roots, edges + 3 * nf);
    }
    if (nc < 1 || (nc > 1 && (int64_t)h != nc)) {  // a forest over n points in nc components
        set_error("kruskal: %lld forest edges for %lld points in %lld components", (long long)nf,
                  (long long)n, (long long)(nc < 1 ? nc : (int64_t)h));
        return FHG_ERR_NO_CONVERGENCE;
    }
    *n_components = nc;
    return FHG_OK;
}

}  // namespace fhg
