// Boruvka minimum spanning tree over mutual reachability, on the GPU.
//
// Replaces boruvka.py:474-647 (initialize_boruvka_from_knn,
// update_component_vectors, boruvka_tree_query, merge_components,
// parallel_boruvka).  Weights are squared float32 mutual-reachability
// distances max(rdist(p, q), core2[p], core2[q]) until the final sqrt.
//
// Round 0 (boruvka.py:474): every point p links to its first kNN neighbour q
// (position >= 1) with core2[p] >= core2[q], weight max(core2[p], rdist).
// These links form a forest except for cycles through equal core distances;
// the reference unions them in point order, so on every cycle the link of
// the largest point index is the one it skips -- dropped here the same way.
//
// Round r >= 1: for every point, the best edge to another component by
// (weight, caller index of the far end), found by a warp-cooperative walk of
// the bucket tree that skips nodes lying wholly inside the point's own
// component (node_comp, boruvka.py:98-124) and nodes beyond the component's
// running bound (boruvka.py:182-186).  Each component keeps its minimum in a
// 64-bit word (weight bits << 32 | min endpoint index) updated by atomicMin,
// with a second 32-bit atomicMin on the max endpoint index: together the
// total order (weight, min index, max index).  Under a total order two
// components can only choose each other with the same edge; the edge is
// then written once, oriented from the component whose lowest point index
// is smaller -- the component the reference's merge loop visits first.
// Components merge with a lock-free union-find; edges of a round are written
// in order of each component's lowest point index (the reference's dict
// insertion order).
#include "compact.cuh"
#include "mst.cuh"
#include "radius.cuh"
#include "primitives.cuh"
#include "reftree.cuh"
#include "uf.cuh"

#include <memory>

namespace fhg {
namespace {

constexpr int kSW = 4;        // warps per block, search kernel
// A round's search runs on a list of the searching points when they are fewer
// than kSparseNum / kSparseDen of all points.
constexpr int64_t kSparseNum = 1, kSparseDen = 4;
constexpr int kStack = 64;
constexpr int kMaxRounds = 64;
// Levels that a dense search expands at once (32 nodes, one per lane), and its
// stack: 31 nodes wait at every expanded depth of at most 26 / 5.
constexpr int kWideLevels = 5, kWideStack = 6 * 32;
constexpr int32_t kEmpty = -2;  // node_comp of a node with no points
constexpr int32_t kMixed = -1;  // node_comp of a node spanning components

__device__ __forceinline__ unsigned long long pack_key(float w, int32_t lo) {
    return ((unsigned long long)__float_as_uint(w) << 32) | (uint32_t)lo;
}
__device__ __forceinline__ float key_weight(unsigned long long k) {
    return __uint_as_float((uint32_t)(k >> 32));
}

// ------------------------------------------------------------- kNN to core
// core2 = squared distance to the k-th neighbour (itself included); +inf when
// there are fewer than k points, 0 for min_samples <= 1 (boruvka.py:581-601).
// open[p] arrives as the kNN kernel's boundary-tie flag and leaves as "a seed
// of weight core2[p] is not provably final": some point outside p's list may
// lie within core2[p] in squared distance (the core value passes the list's
// k-th squared distance, or reaches it while another point ties with it).
__device__ __forceinline__ int8_t seed_open(float c, float kth, int8_t tie) {
    return (!(c < kth) && (c > kth || tie)) ? 1 : 0;
}
__device__ __forceinline__ void core_body(int64_t p, int kk, int k, int ms, const float* knn_d_s,
                                          float* core2, int8_t* open) {
    const float kth = knn_d_s[p * kk + kk - 1];
    const float c = ms <= 1 ? 0.0f : (k > kk ? INFINITY : kth);
    core2[p] = c;
    open[p] = seed_open(c, kth, open[p]);
}

// Weighted core distance (boruvka.py:527 sample_weight_core_distance): the
// plain distance (sqrt of the squared one, boruvka.py:563 queries without
// output_rdist) to the first neighbour at which the running weight, the
// point's own included, reaches min_samples.  Slots past the list are the
// reference's padding (+inf, index -1 -> the weight of the last point).
__global__ void weighted_core_kernel(int64_t n, int kk, int kq, int ms,
                                     const float* __restrict__ knn_d_s,
                                     const int32_t* __restrict__ knn_s,
                                     const float* __restrict__ w_s, float w_last,
                                     float* __restrict__ core2, int8_t* __restrict__ open) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    double total = 0.0;
    int j = 0;
    while (total < (double)ms && j < kq) {
        const int32_t q = j < kk ? knn_s[p * kk + j] : -1;
        total += (double)(q >= 0 ? w_s[q] : w_last);
        ++j;
    }
    const int jj = j > 0 ? j - 1 : kq - 1;
    const float c = jj < kk ? __fsqrt_rn(knn_d_s[p * kk + jj]) : INFINITY;
    core2[p] = c;
    open[p] = seed_open(c, knn_d_s[p * kk + kk - 1], open[p]);
}
__global__ void gather_weights_kernel(int64_t n, const int32_t* __restrict__ orig,
                                      const float* __restrict__ w, float* __restrict__ w_s) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) w_s[p] = w[orig[p]];
}

// Core distances in caller order; neighbour columns past the kNN list (the
// reference's padding when k exceeds the point count) are -1.  The kNN kernel
// writes the other neighbour columns itself.
__device__ __forceinline__ void outputs_body(int64_t p, int kk, int k, const int32_t* orig,
                                             const float* core2, float* core_o, int32_t* nbr_o) {
    const int64_t o = orig[p];
    if (core_o) core_o[o] = __fsqrt_rn(core2[p]);
    if (nbr_o)
        for (int j = kk > 1 ? kk : 1; j < k; ++j) nbr_o[o * (k - 1) + j - 1] = -1;
}
// core_from_knn: the unweighted core distances first.
__global__ void core_outputs_kernel(int64_t n, int kk, int k, int ms, int core_from_knn,
                                    const float* __restrict__ knn_d_s, float* core2,
                                    int8_t* open, const int32_t* __restrict__ orig, float* core_o,
                                    int32_t* nbr_o) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    if (core_from_knn) core_body(p, kk, k, ms, knn_d_s, core2, open);
    outputs_body(p, kk, k, orig, core2, core_o, nbr_o);
}

// ------------------------------------------------------- state of the rounds
// Everything a round reads and writes, in index order unless noted.  The
// bodies below take it by value and are run by one kernel each, or -- for few
// points, where the launches themselves are the time -- one after the other
// inside a single block (small_*_kernel).  No pointer is __restrict__: a block
// reads what it wrote a barrier earlier.
// Counts and flags kept on the device: edges and components so far, edges of
// the round, flags, rounds and the components at the start of each.
enum : int { kStEdges = 0, kStComps, kStAdded, kStMissing, kStEqual, kStRounds, kStHistory };
constexpr int kStWords = kStHistory + kMaxRounds;
struct BorState {
    int64_t n, nleaves, slots;
    int k, ref_ties, plain_d;
    const int32_t *orig, *rank;
    const float* knn_d;
    const int32_t* knn_s;
    float* core2;
    int32_t *target, *par, *comp;  // par: union-find over points, then components
    float* w0;
    // cmin: a component's lowest caller index.  The components in its order
    // (the reference's dict order): representative and cmin; next round's.
    int32_t *cmin, *reps, *rep_cmin, *next_reps, *next_cmin;
    unsigned long long* keyA;
    uint32_t* keyB;
    int32_t *winner, *tgt;
    float* cand_w;
    int32_t* cand_q;
    int8_t* exhausted;
    int2* nc;
    int32_t *src, *dst;
    float* w2;
    uint32_t* stat;  // [kStWords]
};

// ----------------------------------------------------------------- round 0
// plain_d: the weighted path's round 0 works on plain (not squared) distances.
__device__ __forceinline__ void round0_body(const BorState& S, int64_t p) {
    const int k = S.k;
    const float cp = S.core2[p];
    int32_t t = -1;
    float w = 0.0f;
    for (int j = 1; j < k; ++j) {
        const int32_t q = S.knn_s[p * k + j];
        if (q < 0) break;
        const float cq = S.core2[q];
        if (cp >= cq) {
            if (q != p) {
                t = q;
                const float d = S.knn_d[p * k + j];
                w = fmaxf(cp, S.plain_d ? __fsqrt_rn(d) : d);
                if (cq == cp) S.stat[kStEqual] = 1u;
            }
            break;
        }
    }
    S.target[p] = t;
    S.w0[p] = w;
    S.par[p] = (int32_t)p;
    S.cmin[p] = INT32_MAX;
    S.cand_q[p] = -1;  // no candidate yet
    S.exhausted[p] = 0;
}
__global__ void round0_kernel(BorState S) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) round0_body(S, p);
}

__device__ __forceinline__ void union_target_body(const BorState& S, int64_t p) {
    const int32_t t = S.target[p];
    if (t >= 0) uf_union(S.par, (int32_t)p, t);
}
__global__ void union_targets_kernel(BorState S) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) union_target_body(S, p);
}
__device__ __forceinline__ void flatten_body(const BorState& S, int64_t p) {
    const int32_t c = uf_find(S.par, (int32_t)p);
    S.comp[p] = c;
    // most points find their component's minimum already at or below theirs
    const int32_t o = S.orig[p];
    if (o < *(volatile int32_t*)&S.cmin[c]) atomicMin(&S.cmin[c], o);
}
__global__ void flatten_kernel(BorState S) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) flatten_body(S, p);
}

// Functional-graph cycle detection by pointer doubling (only run when some
// round-0 link joins two equal core distances).
__device__ __forceinline__ void cyc_init_body(const BorState& S, int64_t p, int32_t* nxt,
                                              int32_t* mx) {
    nxt[p] = S.target[p] >= 0 ? S.target[p] : (int32_t)p;
    mx[p] = S.orig[p];
}
__global__ void cyc_init_kernel(BorState S, int32_t* nxt, int32_t* mx) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) cyc_init_body(S, p, nxt, mx);
}
// `changed` (nullable) is set when some node's window maximum grew.  A step
// that grows none has converged: every node's maximum is then at least the
// next window's, and by induction the maximum over all it reaches.
__global__ void cyc_step_kernel(int64_t n, const int32_t* __restrict__ nxt,
                                const int32_t* __restrict__ mx, int32_t* __restrict__ nxt2,
                                int32_t* __restrict__ mx2, int* __restrict__ changed) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int32_t q = nxt[p];
    nxt2[p] = nxt[q];
    const int32_t a = mx[p], b = mx[q];
    mx2[p] = max(a, b);
    if (changed && b > a) *changed = 1;
}
__device__ __forceinline__ void cyc_drop_body(const BorState& S, int64_t p, const int32_t* nxt,
                                              const int32_t* mx) {
    if (S.target[p] >= 0 && mx[nxt[p]] == S.orig[p]) S.target[p] = -1;
}
__global__ void cyc_drop_kernel(BorState S, const int32_t* nxt, const int32_t* mx) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) cyc_drop_body(S, p, nxt, mx);
}

// Round-0 edges, by caller index of the choosing point (the reference's
// order), or in index order when the order does not matter.
struct Round0Edges {
    BorState S;
    int by_caller;
    __device__ int32_t point(int64_t i) const { return by_caller ? S.rank[i] : (int32_t)i; }
    __device__ bool test(int64_t i) const { return S.target[point(i)] >= 0; }
    __device__ void emit(int64_t i, uint32_t at) const {
        const int32_t p = point(i);
        S.src[at] = S.orig[p];
        S.dst[at] = S.orig[S.target[p]];
        S.w2[at] = S.w0[p];
    }
    __device__ void each(int64_t) const {}
};

__device__ __forceinline__ void reset_component(const BorState& S, int32_t c) {
    S.keyA[c] = ~0ull;
    S.keyB[c] = 0xffffffffu;
    S.winner[c] = -1;
}
// The components in the order of their lowest caller index i.
struct FirstComponents {
    BorState S;
    __device__ bool test(int64_t i) const { return S.cmin[S.comp[S.rank[i]]] == (int32_t)i; }
    __device__ void emit(int64_t i, uint32_t at) const {
        const int32_t c = S.comp[S.rank[i]];
        S.reps[at] = c;
        S.rep_cmin[at] = (int32_t)i;
        reset_component(S, c);
    }
    __device__ void each(int64_t) const {}
};

// ---------------------------------------------------------- per round: nodes
// Per node: x = its single component (node_comp, boruvka.py:98-124), kMixed
// or kEmpty; y = bits of the least core distance of its points.  Every edge
// into the node weighs at least that core distance, so a node whose least
// core distance exceeds a query's threshold is skipped like a distant one.
// The kernels cover the tree in pieces: a block joins the kNodeLeaves leaves of
// its chunk up to the chunk's root, then blocks of kNodeTop nodes go on.  A
// leaf's points take their new component first (relabel).
constexpr int kNodeLeaves = 64, kNodeThreads = 256, kNodeTop = 512;
__device__ __forceinline__ void leaf_node_body(const BorState& S, int64_t leaf, int lane,
                                               int relabel) {
    const int64_t i = leaf * kLeaf + lane;
    const bool valid = leaf < S.nleaves && i < S.n;
    int32_t c = 0;
    if (valid) {
        c = S.comp[i];
        if (relabel) {
            c = uf_find(S.par, c);
            S.comp[i] = c;
        }
    }
    // non-negative floats order like their bit patterns
    int32_t kb = valid ? __float_as_int(S.core2[i]) : INT32_MAX;
    const int32_t c0 = __shfl_sync(kFull, c, 0);
    const bool same = __all_sync(kFull, !valid || c == c0);
    kb = __reduce_min_sync(kFull, kb);
    if (lane == 0)
        S.nc[S.slots - 1 + leaf] =
            make_int2(leaf >= S.nleaves ? kEmpty : (same ? c0 : kMixed), kb);
}
__device__ __forceinline__ void join_node_body(int2* nc, int64_t node) {
    const int2 l = nc[2 * node + 1], r = nc[2 * node + 2];
    nc[node] = make_int2(l.x == kEmpty ? r.x : (r.x == kEmpty ? l.x : (l.x == r.x ? l.x : kMixed)),
                         min(l.y, r.y));
}
__global__ void __launch_bounds__(kNodeThreads) node_chunk_kernel(BorState S, int relabel) {
    const int leaves = (int)min(S.slots, (int64_t)kNodeLeaves);
    for (int l = threadIdx.x >> 5; l < leaves; l += kNodeThreads / 32)
        leaf_node_body(S, (int64_t)blockIdx.x * kNodeLeaves + l, threadIdx.x & 31, relabel);
    int64_t level = S.slots - 1;
    for (int width = leaves / 2; width >= 1; width >>= 1) {
        __syncthreads();
        level = (level - 1) / 2;
        if (threadIdx.x < width)
            join_node_body(S.nc, level + (int64_t)blockIdx.x * width + threadIdx.x);
    }
}
__global__ void __launch_bounds__(kNodeTop / 2) node_top_kernel(int2* nc, int64_t width) {
    const int span = (int)min(width, (int64_t)kNodeTop);
    int64_t level = width - 1;
    for (int wd = span / 2; wd >= 1; wd >>= 1) {
        level = (level - 1) / 2;
        if (threadIdx.x < wd) join_node_body(nc, level + (int64_t)blockIdx.x * wd + threadIdx.x);
        __syncthreads();
    }
}

// ------------------------------------------------------- per round: seeds
// Every point's best edge among its own kNN list (boruvka.py:474 uses the same
// lists), published to its component's key before any point searches, so the
// search starts from every component's seed bound.
// exhausted[p]: every kNN neighbour of p was already in p's component in an
// earlier round -- it stays so, as components only merge.
__device__ __forceinline__ void seed_body(const BorState& S, int64_t p) {
    const int k = S.k;
    const int32_t c = S.comp[p];
    // The previous round's candidate of this point is still an edge out of
    // its component when its target has not been merged in: it seeds the
    // point's best (when it beats the kNN seed) and its component's key
    // before any point searches.  The search still finds every edge within
    // that bound, so the point's final candidate is its exact best.  (Its
    // weight equals the core distance only for a target inside the kNN
    // radius, which the kNN seed has already met, so the seed-finality rule
    // below is unaffected.)
    const int32_t oq = S.cand_q[p];
    const float ow = S.cand_w[p];
    const int32_t oo = (oq >= 0 && S.comp[oq] != c) ? S.orig[oq] : -1;
    float bw = INFINITY;
    int32_t bq = -1, bo = INT32_MAX;
    if (!S.exhausted[p]) {
        const float cp = S.core2[p];
        // kSeedAhead neighbours and their components are read together: one at
        // a time, each waited for two gathers (10M points, k = 16, all rounds:
        // 2.12 -> 2.07 ms; 2M x 5-D, k = 11: 381 -> 318 us; 300k, k = 101: 417 -> 286)
        constexpr int kSeedAhead = 4;
        for (int j = 1; j < k; j += kSeedAhead) {
            int32_t qs[kSeedAhead], cq[kSeedAhead];
#pragma unroll
            for (int u = 0; u < kSeedAhead; ++u)
                qs[u] = j + u < k ? S.knn_s[p * k + j + u] : -1;
#pragma unroll
            for (int u = 0; u < kSeedAhead; ++u) cq[u] = qs[u] >= 0 ? S.comp[qs[u]] : c;
#pragma unroll
            for (int u = 0; u < kSeedAhead; ++u) {
                if (cq[u] == c) continue;
                const float w = fmaxf(fmaxf(S.knn_d[p * k + j + u], cp), S.core2[qs[u]]);
                const int32_t o = S.orig[qs[u]];
                if (w < bw || (w == bw && o < bo)) {
                    bw = w;
                    bq = qs[u];
                    bo = o;
                }
            }
            if (qs[kSeedAhead - 1] < 0) break;  // (an empty slot: the list ends)
        }
        if (bq < 0) S.exhausted[p] = 1;  // no other component in the kNN list
    }
    if (oo >= 0 && (ow < bw || (ow == bw && oo < bo))) {
        bw = ow;
        bq = oq;
        bo = oo;
    }
    S.cand_w[p] = bw;
    S.cand_q[p] = bq;
    if (bq >= 0) {
        const unsigned long long key =
            pack_key(bw, S.ref_ties ? S.orig[p] : min(S.orig[p], bo));
        if (key < *(volatile unsigned long long*)&S.keyA[c]) atomicMin(&S.keyA[c], key);
    }
}
__global__ void seed_kernel(BorState S) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) seed_body(S, p);
}

// ------------------------------------------------------- per round: search
// A node is entered when some lane's point lies outside the node's single
// component (node_comp) and within that lane's threshold -- the smaller of its
// own best weight and its component's running best (boruvka.py:182-191).
//
// A point whose seed already weighs its own core distance (the least weight
// any of its edges can have) is settled without a search when every point
// at that distance is in its kNN list: the core distance is below the k-th
// distance, or no point outside the list lies exactly at the k-th distance
// (knn_open clear).  Any other edge then weighs more than the seed.

// Order-preserving map of float bits to uint32, and back.
__device__ __forceinline__ uint32_t ordered_bits(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float ordered_float(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? u & 0x7fffffffu : ~u);
}

// One warp's searching points (one per lane) and a bucket scan for them.
template <int DIM, int SP>
struct Searcher {
    const IndexView& ix;
    const float* core2;
    const int32_t* comp;
    unsigned long long* keyA;
    float4* xyz;     // [32 * SP / 4] a bucket's points
    float4* queries; // [32 * SP / 4] the lanes' points
    int2* cc;        // [32] (component, core bits) of the bucket
    int32_t* co;     // [32] caller indices of the bucket
    int lane;
    float q[DIM];
    int32_t c;       // this lane's component
    float cp, bw;    // core distance, best weight so far
    int32_t bq, bo;  // its far end: index position, caller index
    float thr;       // min(bw, the component's running best)
    bool active;

    __device__ __forceinline__ void refresh() {
        if (active) {
            thr = fminf(thr, key_weight(*(volatile unsigned long long*)&keyA[c]));
            active = !(cp > thr);
        }
    }

    // The bucket's candidates for the lanes that need it.  Only candidates
    // that can matter to some needing lane are considered: a core distance
    // within the largest needing threshold, and -- when every needing lane is
    // in one component -- outside it.  The best edge is a minimum over
    // (weight, index), so the order of the visits does not change it.  Few
    // needing lanes take the candidates one per lane and a warp minimum each;
    // otherwise every candidate is read by all of them.
    __device__ __forceinline__ void scan(int64_t lf, bool need) {
        const int64_t base = lf * kLeaf;
        const int cnt = (int)(ix.n - base < kLeaf ? ix.n - base : kLeaf);
        float own[SP];
        int2 mine = make_int2(0, 0);
        int32_t own_o = 0;
#pragma unroll
        for (int j = 0; j < SP; ++j) own[j] = 0.0f;
        if (lane < cnt) {
            load_pt<SP>(ix.pts, base + lane, own);
            mine = make_int2(comp[base + lane], __float_as_int(core2[base + lane]));
            own_o = ix.orig[base + lane];
        }
        const unsigned needers = __ballot_sync(kFull, need);
        const float mthr =
            __uint_as_float(__reduce_max_sync(kFull, need ? __float_as_uint(thr) : 0u));
        const int32_t c0 = __shfl_sync(kFull, c, __ffs(needers) - 1);
        const bool one_comp = __all_sync(kFull, !need || c == c0);
        const bool relevant =
            lane < cnt && !(__int_as_float(mine.y) > mthr) && !(one_comp && mine.x == c0);
        unsigned todo = __ballot_sync(kFull, relevant);
        if (!todo) {
            refresh();
            return;
        }
        if (2 * __popc(needers) <= __popc(todo)) {
            const float core = __int_as_float(mine.y);
            for (unsigned m = needers; m; m &= m - 1u) {
                const int i = __ffs(m) - 1;
                float y[SP];
#pragma unroll
                for (int h = 0; h < SP / 4; ++h) {
                    const float4 v = queries[i * (SP / 4) + h];
                    y[4 * h] = v.x; y[4 * h + 1] = v.y; y[4 * h + 2] = v.z; y[4 * h + 3] = v.w;
                }
                const float cpi = __shfl_sync(kFull, cp, i), bwi = __shfl_sync(kFull, bw, i);
                const int32_t ci = __shfl_sync(kFull, c, i);
                const float w = fmaxf(fmaxf(rdist_rn<DIM>(y, own), cpi), core);
                const bool in = relevant && mine.x != ci && w <= bwi;
                if (!__any_sync(kFull, in)) continue;
                // non-negative floats order like their bits
                const uint32_t wm = __reduce_min_sync(kFull, in ? __float_as_uint(w) : 0xffffffffu);
                const bool low = in && __float_as_uint(w) == wm;
                const uint32_t om = __reduce_min_sync(kFull, low ? (uint32_t)own_o : 0xffffffffu);
                const int t = __ffs(__ballot_sync(kFull, low && (uint32_t)own_o == om)) - 1;
                if (lane == i) {
                    const float wl = __uint_as_float(wm);
                    if (wl < bw || (int32_t)om < bo) {
                        bw = wl;
                        bq = (int32_t)(base + t);
                        bo = (int32_t)om;
                        thr = fminf(thr, bw);
                    }
                }
            }
        } else {
            __syncwarp();
            if (lane < cnt) {
#pragma unroll
                for (int h = 0; h < SP / 4; ++h)
                    xyz[lane * (SP / 4) + h] =
                        make_float4(own[4 * h], own[4 * h + 1], own[4 * h + 2], own[4 * h + 3]);
                cc[lane] = mine;
                co[lane] = own_o;
            }
            __syncwarp();
            for (; todo; todo &= todo - 1u) {
                const int t = __ffs(todo) - 1;
                const int2 tcc = cc[t];
                const float tk = __int_as_float(tcc.y);
                if (need && tcc.x != c && tk <= thr) {
                    float x[SP];
#pragma unroll
                    for (int h = 0; h < SP / 4; ++h) {
                        const float4 v = xyz[t * (SP / 4) + h];
                        x[4 * h] = v.x; x[4 * h + 1] = v.y; x[4 * h + 2] = v.z; x[4 * h + 3] = v.w;
                    }
                    const float w = fmaxf(fmaxf(rdist_rn<DIM>(q, x), cp), tk);
                    if (w <= bw) {
                        const int32_t to = co[t];
                        if (w < bw || to < bo) {
                            bw = w;
                            bq = (int32_t)(base + t);
                            bo = to;
                            thr = fminf(thr, bw);
                        }
                    }
                }
            }
        }
        refresh();
    }
};

// Few points search: a warp takes 32 consecutive entries of a list of them (in
// index order) and walks from the root, children of least bound over its
// lanes first; both children are tested when their parent is expanded.
// Many points search: a warp takes a bucket, and its lanes test up to 32 nodes
// at once -- the descendants five levels down -- against the box and the
// largest threshold of the bucket's searching points: no bound of a single
// point to a node is below the bound between the two boxes (every operation
// rounds monotonically).  A node left over is expanded in turn, a bucket left
// over gets a test per lane before it is scanned.  (One node after another,
// every lane testing its own point, took two thirds of this kernel's
// instructions.)  pass 0 stays inside the 32 buckets around the home bucket,
// pass 1 takes the others, so that every component's bound from its nearby
// candidates is published before any point searches far away; pass 2 is both.
// `split` warps share a bucket's (or 32 list entries') points, 32 / split each.
template <int DIM, int SP>
__global__ void __launch_bounds__(kSW * 32) search_kernel(
    IndexView ix, const int8_t* __restrict__ knn_open, const float* __restrict__ core2,
    const int32_t* __restrict__ comp, const int2* __restrict__ nc, unsigned long long* keyA,
    float* __restrict__ cand_w, int32_t* __restrict__ cand_q, int pass,
    const int32_t* __restrict__ plist, int64_t plen, int ref_ties, int split,
    const uint32_t* __restrict__ stat) {
    __shared__ int32_t s_stack[kSW][kWideStack];
    __shared__ float4 s_xyz[kSW][32 * (SP / 4)], s_q[kSW][32 * (SP / 4)];
    __shared__ int2 s_cc[kSW][32];
    __shared__ int32_t s_orig[kSW][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool sparse = plist != nullptr;
    const int64_t part = (int64_t)blockIdx.x * kSW + warp;
    const int64_t leaf = part / split;
    if (sparse ? leaf * 32 >= plen : leaf >= ix.nleaves) return;
    if (stat[kStComps] <= 1) return;  // (a round launched after the last)
    const int64_t li = leaf * 32 + lane;
    const int64_t p = sparse ? (li < plen ? plist[li] : 0) : leaf * kLeaf + lane;
    const bool valid =
        lane * split / 32 == (int)(part % split) && (sparse ? li < plen : p < ix.n);
    Searcher<DIM, SP> S{ix, core2, comp, keyA, s_xyz[warp], s_q[warp], s_cc[warp], s_orig[warp],
                        lane};
    S.c = -3;
    S.cp = 0.0f;
    S.bw = INFINITY;
    S.bq = -1;
    S.bo = INT32_MAX;
    S.active = false;
    S.thr = INFINITY;
    if (valid) {
        S.c = comp[p];
        S.cp = core2[p];
        S.bw = cand_w[p];
        S.bq = cand_q[p];
        if (S.bq >= 0) S.bo = ix.orig[S.bq];
        const bool settled = S.bq >= 0 && S.bw == S.cp && !knn_open[p];
        S.thr = fminf(S.bw, key_weight(*(volatile unsigned long long*)&keyA[S.c]));
        S.active = !settled && !(S.cp > S.thr);
    }
    if (!__any_sync(kFull, S.active)) return;
    const int32_t seed_q = S.bq;
    {
        float t[SP];
#pragma unroll
        for (int j = 0; j < SP; ++j) t[j] = 0.0f;
        if (valid) load_pt<SP>(ix.pts, p, t);
#pragma unroll
        for (int j = 0; j < DIM; ++j) S.q[j] = t[j];
#pragma unroll
        for (int h = 0; h < SP / 4; ++h)
            s_q[warp][lane * (SP / 4) + h] =
                make_float4(t[4 * h], t[4 * h + 1], t[4 * h + 2], t[4 * h + 3]);
    }
    __syncwarp();
    int32_t* st = s_stack[warp];
    const int64_t first_leaf_node = ix.slots - 1;
    auto other = [&](int2 ncn) { return ncn.x != S.c && ncn.x != kEmpty; };
    if (sparse) {
        // A lane's key for a node is max(box bound, least core) when the node
        // holds points of another component; the node is needed when the key
        // is within the lane's threshold.
        auto key_of = [&](int2 ncn, const float* b) {
            return other(ncn) ? fmaxf(box_lb_n<DIM, SP>(b, S.q), __int_as_float(ncn.y)) : INFINITY;
        };
        float b0[2 * SP];
        load_box<SP>(ix.box, 0, b0);
        int sp = 0;
        if (__any_sync(kFull, S.active && key_of(nc[0], b0) <= S.thr)) {
            if (first_leaf_node == 0) {
                S.scan(0, S.active && key_of(nc[0], b0) <= S.thr);
            } else {
                if (lane == 0) st[0] = 0;
                sp = 1;
            }
        }
        __syncwarp();
        while (sp > 0) {
            --sp;
            const int32_t node = st[sp];
            __syncwarp();
            const int32_t l = 2 * node + 1, r = l + 1;
            const int2 ncl = nc[l], ncr = nc[r];
            bool nl = S.active && other(ncl) && !(__int_as_float(ncl.y) > S.thr);
            bool nr = S.active && other(ncr) && !(__int_as_float(ncr.y) > S.thr);
            if (!__any_sync(kFull, nl || nr)) continue;
            float bl[2 * SP], br[2 * SP];
            load_box<SP>(ix.box, l, bl);
            load_box<SP>(ix.box, r, br);
            const float kl = key_of(ncl, bl), kr = key_of(ncr, br);
            nl = nl && kl <= S.thr;
            nr = nr && kr <= S.thr;
            const bool al = __any_sync(kFull, nl), ar = __any_sync(kFull, nr);
            if (!al && !ar) continue;
            bool left_first = al;
            if (al && ar)  // non-negative floats order like their bits
                left_first = __reduce_min_sync(kFull, nl ? __float_as_uint(kl) : 0x7f800000u) <=
                             __reduce_min_sync(kFull, nr ? __float_as_uint(kr) : 0x7f800000u);
            if (l >= first_leaf_node) {
                // thresholds may shrink while the first bucket is scanned
                for (int turn = 0; turn < 2; ++turn) {
                    const bool left = left_first == (turn == 0);
                    const bool need = S.active && (left ? kl : kr) <= S.thr;
                    if (__any_sync(kFull, need)) S.scan((left ? l : r) - first_leaf_node, need);
                }
            } else {
                if (lane == 0) {
                    int t = sp;
                    if (left_first ? ar : al) st[t++] = left_first ? r : l;
                    st[t] = left_first ? l : r;
                }
                sp += al && ar ? 2 : 1;
                __syncwarp();
            }
        }
    } else {
        // One component after another: its searching points' box and largest
        // threshold.  (Two components of one bucket can have thresholds far
        // apart, and only the nodes that lie wholly inside the searching
        // component fall away early.)
        bool pending = S.active;
        for (unsigned pm = __ballot_sync(kFull, pending); pm;
             pm = __ballot_sync(kFull, pending)) {
            const int32_t c0 = __shfl_sync(kFull, S.c, __ffs(pm) - 1);
            S.active = pending && S.c == c0;
            pending = pending && S.c != c0;
            S.refresh();
            if (!__any_sync(kFull, S.active)) continue;
            float qlo[DIM], qhi[DIM];
#pragma unroll
            for (int j = 0; j < DIM; ++j) {
                const uint32_t u = ordered_bits(S.q[j]);
                qlo[j] = ordered_float(__reduce_min_sync(kFull, S.active ? u : 0xffffffffu));
                qhi[j] = ordered_float(__reduce_max_sync(kFull, S.active ? u : 0u));
            }
            auto largest_thr = [&]() {
                return __uint_as_float(
                    __reduce_max_sync(kFull, S.active ? __float_as_uint(S.thr) : 0u));
            };
            float T = largest_thr();
            // Lane's node against the points' box; NaN for a node to leave out (+inf is
            // a bound like any other: squared distances overflow, core distances
            // are infinite where there are fewer points than neighbours).
            auto box_key = [&](int64_t node, int2 ncn) {
                if (ncn.x == kEmpty || ncn.x == c0 || __int_as_float(ncn.y) > T) return NAN;
                float b[2 * SP];
                load_box<SP>(ix.box, node, b);
                float r = 0.0f;
#pragma unroll
                for (int j = 0; j < DIM; ++j) {
                    const float dd =
                        fmaxf(fmaxf(__fsub_rn(b[j], qhi[j]), __fsub_rn(qlo[j], b[SP + j])), 0.0f);
                    r = __fadd_rn(r, __fmul_rn(dd, dd));
                }
                return fmaxf(r, __int_as_float(ncn.y));
            };
            const int depth = 63 - __clzll(ix.slots);  // of the buckets
            const int64_t home_group = leaf >> kWideLevels;
            // the 32 buckets from 32 * group on, nearest first
            auto scan_group = [&](int64_t group) {
                const int size = ix.slots < 32 ? (int)ix.slots : 32;
                const int64_t node = first_leaf_node + group * 32 + lane;
                int2 ncn = make_int2(kEmpty, 0);
                float key = NAN;
                if (lane < size) {
                    ncn = nc[node];
                    key = box_key(node, ncn);
                }
                unsigned left = __ballot_sync(kFull, key <= T);
                while (left) {
                    const uint32_t mine = (left >> lane) & 1u ? __float_as_uint(key) : 0xffffffffu;
                    const uint32_t least = __reduce_min_sync(kFull, mine);
                    if (__uint_as_float(least) > T) break;
                    const int t = __ffs(__ballot_sync(kFull, mine == least)) - 1;
                    left &= ~(1u << t);
                    const int64_t lf = group * 32 + t;
                    const float core = __int_as_float(__shfl_sync(kFull, ncn.y, t));
                    bool need = S.active && !(core > S.thr);
                    if (need) {
                        float b[2 * SP];
                        load_box<SP>(ix.box, first_leaf_node + lf, b);
                        need = box_lb_n<DIM, SP>(b, S.q) <= S.thr;
                    }
                    if (!__any_sync(kFull, need)) continue;
                    S.scan(lf, need);
                    T = largest_thr();
                    if (!__any_sync(kFull, S.active)) break;
                }
            };
            if (pass != 1) scan_group(home_group);
            if (pass != 0 && depth > kWideLevels && __any_sync(kFull, S.active)) {
                int sp = 0;
                int64_t node = 0;  // the node to expand
                int at = 0;        // its depth
                for (;;) {
                    const int step =
                        at == 0 && depth % kWideLevels ? depth % kWideLevels : kWideLevels;
                    const int64_t first = ((node + 1) << step) - 1;
                    if (at + step == depth) {
                        const int64_t group = (first - first_leaf_node) >> kWideLevels;
                        if (group != home_group) scan_group(group);
                    } else {
                        const int64_t mine = first + lane;
                        float key = NAN;
                        if (lane < (1 << step)) key = box_key(mine, nc[mine]);
                        const unsigned in = __ballot_sync(kFull, key <= T);
                        if (in) {  // the nearest on top of the stack
                            const bool on = (in >> lane) & 1u;
                            const uint32_t bits = on ? __float_as_uint(key) : 0xffffffffu;
                            const uint32_t least = __reduce_min_sync(kFull, bits);
                            const int top = __ffs(__ballot_sync(kFull, on && bits == least)) - 1;
                            const unsigned rest = in & ~(1u << top);
                            if ((rest >> lane) & 1u)
                                st[sp + __popc(rest & ((1u << lane) - 1u))] = (int32_t)mine;
                            if (lane == top) st[sp + __popc(rest)] = (int32_t)mine;
                            sp += __popc(in);
                            __syncwarp();
                        }
                    }
                    if (sp == 0 || !__any_sync(kFull, S.active)) break;
                    node = st[--sp];
                    at = 63 - __clzll(node + 1);
                    __syncwarp();
                }
            }
        }
    }
    if (!valid || S.bq == seed_q) return;
    cand_w[p] = S.bw;
    cand_q[p] = S.bq;
    const unsigned long long key =
        pack_key(S.bw, ref_ties ? ix.orig[p] : min(ix.orig[p], S.bo));
    if (key < *(volatile unsigned long long*)&keyA[S.c]) atomicMin(&keyA[S.c], key);
}

// The points that start the search searching (as search_kernel decides).
struct SearchingPoints {
    BorState S;
    const int8_t* knn_open;
    int32_t* list;
    __device__ bool test(int64_t p) const {
        const float cp = S.core2[p], bw = S.cand_w[p];
        const bool settled = S.cand_q[p] >= 0 && bw == cp && !knn_open[p];
        const float thr0 = fminf(bw, key_weight(S.keyA[S.comp[p]]));
        return !settled && !(cp > thr0);
    }
    __device__ void emit(int64_t p, uint32_t at) const { list[at] = (int32_t)p; }
    __device__ void each(int64_t) const {}
};

// ---------------------------------------------------- per round: the merge
// Every component's winner: the point that holds its least (weight, lowest
// index) with, among those, the least highest index.
__device__ __forceinline__ void stage_b_body(const BorState& S, int64_t p) {
    const int32_t q = S.cand_q[p];
    if (q < 0) return;
    const int32_t c = S.comp[p], op = S.orig[p], oq = S.orig[q];
    if (S.keyA[c] == pack_key(S.cand_w[p], min(op, oq)))
        atomicMin(&S.keyB[c], (uint32_t)max(op, oq));
}
__device__ __forceinline__ void stage_c_body(const BorState& S, int64_t p) {
    const int32_t q = S.cand_q[p];
    if (q < 0) return;
    const int32_t c = S.comp[p], op = S.orig[p], oq = S.orig[q];
    if (S.keyA[c] == pack_key(S.cand_w[p], min(op, oq)) && S.keyB[c] == (uint32_t)max(op, oq))
        S.winner[c] = (int32_t)p;
}
__global__ void stage_b_kernel(BorState S) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) stage_b_body(S, p);
}
__global__ void stage_c_kernel(BorState S) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < S.n) stage_c_body(S, p);
}

__device__ __forceinline__ void select_body(const BorState& S, int64_t i) {
    const int32_t c = S.reps[i], p = S.winner[c];
    S.tgt[c] = p < 0 ? -1 : S.comp[S.cand_q[p]];
    if (p < 0) S.stat[kStMissing] = 1u;
}
// The round's edges, in the order of the components' lowest caller indices:
// of a pair that chose each other, the first one's.  (In the reference tie
// mode the cycles have been dropped from tgt already.)
struct RoundEdges {
    BorState S;
    __device__ bool test(int64_t i) const {
        const int32_t c = S.reps[i], t = S.tgt[c];
        if (t < 0) return false;
        return S.ref_ties || S.tgt[t] != c || S.cmin[c] < S.cmin[t];
    }
    __device__ void emit(int64_t i, uint32_t at) const {
        const int32_t p = S.winner[S.reps[i]];
        const uint32_t e = S.stat[kStEdges] + at;
        S.src[e] = S.orig[p];
        S.dst[e] = S.orig[S.cand_q[p]];
        S.w2[e] = S.cand_w[p];
    }
    __device__ void each(int64_t i) const {
        const int32_t c = S.reps[i], t = S.tgt[c];
        if (t >= 0) uf_union(S.par, c, t);
    }
};
__device__ __forceinline__ void merge_cmin_body(const BorState& S, int64_t i) {
    const int32_t c = S.reps[i], r = uf_find(S.par, c);
    if (r != c) atomicMin(&S.cmin[r], S.rep_cmin[i]);
}
// The merged components, each at the place of the old one whose cmin it has.
struct MergedComponents {
    BorState S;
    __device__ bool test(int64_t i) const {
        return S.cmin[uf_find(S.par, S.reps[i])] == S.rep_cmin[i];
    }
    __device__ void emit(int64_t i, uint32_t at) const {
        const int32_t r = uf_find(S.par, S.reps[i]);
        S.next_reps[at] = r;
        S.next_cmin[at] = S.rep_cmin[i];
        reset_component(S, r);
    }
    __device__ void each(int64_t) const {}
};
__global__ void select_kernel(BorState S, int64_t ncomp) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ncomp) select_body(S, i);
}
__global__ void merge_cmin_kernel(BorState S, int64_t ncomp) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) S.stat[kStEdges] += S.stat[kStAdded];
    if (i < ncomp) merge_cmin_body(S, i);
}

// ------------------------------------------------- phases inside one block
// compact() by one block.
template <class F>
__device__ __forceinline__ uint32_t block_compact(const F& f, int64_t n) {
    __shared__ uint32_t s_warp[33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t base = 0;
    for (int64_t i0 = 0; i0 < n; i0 += blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        const bool on = i < n && f.test(i);
        const unsigned b = __ballot_sync(kFull, on);
        if (lane == 0) s_warp[w] = __popc(b);
        __syncthreads();
        if (w == 0) {
            const uint32_t v = lane < nw ? s_warp[lane] : 0u;
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, o);
                if (lane >= o) x += y;
            }
            if (lane < nw) s_warp[lane] = x - v;
            if (lane == 31) s_warp[32] = x;
        }
        __syncthreads();
        if (on) f.emit(i, base + s_warp[w] + __popc(b & ((1u << lane) - 1u)));
        if (i < n) f.each(i);
        base += s_warp[32];
        __syncthreads();
    }
    return base;
}
// From tgt to the merged components (kStEdges, kStComps and the list updated).
__device__ __forceinline__ void block_merge(const BorState& S, int64_t ncomp) {
    const uint32_t added = block_compact(RoundEdges{S}, ncomp);
    for (int64_t i = threadIdx.x; i < ncomp; i += blockDim.x) merge_cmin_body(S, i);
    __syncthreads();
    const uint32_t left = block_compact(MergedComponents{S}, ncomp);
    if (threadIdx.x == 0) {
        S.stat[kStEdges] += added;
        S.stat[kStComps] = left;
        S.stat[kStAdded] = added;
    }
    for (int64_t i = threadIdx.x; i < left; i += blockDim.x) {
        S.reps[i] = S.next_reps[i];
        S.rep_cmin[i] = S.next_cmin[i];
    }
    __syncthreads();
}
constexpr int kSmallThreads = 1024;
// Components of one round that a single block merges in one launch.
constexpr int64_t kBlockMerge = 8192;
__global__ void __launch_bounds__(kSmallThreads) merge_kernel(BorState S, int64_t ncomp) {
    if (!S.ref_ties)
        for (int64_t i = threadIdx.x; i < ncomp; i += blockDim.x) select_body(S, i);
    __syncthreads();
    block_merge(S, ncomp);
}

// Few points: whole phases in one block.  A launch costs about 2 us however
// little it does, the host's read of a count 12 us; a phase over 8,192 points
// costs one block a microsecond or two.
constexpr int64_t kSmallPoints = 8192, kSmallEntries = 32 * 8192;  // points, list entries
__device__ __forceinline__ void block_nodes_and_seeds(const BorState& S, int relabel) {
    for (int64_t l = threadIdx.x >> 5; l < S.slots; l += blockDim.x >> 5)
        leaf_node_body(S, l, threadIdx.x & 31, relabel);
    __syncthreads();
    for (int64_t width = S.slots / 2; width >= 1; width /= 2) {
        for (int64_t t = threadIdx.x; t < width; t += blockDim.x)
            join_node_body(S.nc, width - 1 + t);
        __syncthreads();
    }
    for (int64_t p = threadIdx.x; p < S.n; p += blockDim.x) seed_body(S, p);
}
// Core distances and outputs (as core_outputs_kernel), round 0, and the nodes
// and seeds of round 1.
__global__ void __launch_bounds__(kSmallThreads) small_round0_kernel(
    BorState S, int kq, int ms, int core_from_knn, int8_t* open, float* core_o, int32_t* nbr_o,
    int by_caller, int32_t* nxt, int32_t* mx, int32_t* nxt2, int32_t* mx2) {
    const int64_t n = S.n;
    if (threadIdx.x < kStWords) S.stat[threadIdx.x] = 0u;
    for (int64_t p = threadIdx.x; p < n; p += blockDim.x) {
        if (core_from_knn) core_body(p, S.k, kq, ms, S.knn_d, S.core2, open);
        outputs_body(p, S.k, kq, S.orig, S.core2, core_o, nbr_o);
    }
    __syncthreads();
    for (int64_t p = threadIdx.x; p < n; p += blockDim.x) round0_body(S, p);
    __syncthreads();
    if (S.stat[kStEqual]) {
        for (int64_t p = threadIdx.x; p < n; p += blockDim.x) cyc_init_body(S, p, nxt, mx);
        __syncthreads();
        for (bool grew = true; grew;) {
            bool more = false;
            for (int64_t p = threadIdx.x; p < n; p += blockDim.x) {
                const int32_t q = nxt[p], a = mx[p], b = mx[q];
                nxt2[p] = nxt[q];
                mx2[p] = max(a, b);
                more |= b > a;
            }
            grew = __syncthreads_or(more);
            int32_t* t = nxt; nxt = nxt2; nxt2 = t;
            t = mx; mx = mx2; mx2 = t;
        }
        for (int64_t p = threadIdx.x; p < n; p += blockDim.x) cyc_drop_body(S, p, nxt, mx);
        __syncthreads();
    }
    const uint32_t edges = block_compact(Round0Edges{S, by_caller}, n);
    for (int64_t p = threadIdx.x; p < n; p += blockDim.x) union_target_body(S, p);
    __syncthreads();
    for (int64_t p = threadIdx.x; p < n; p += blockDim.x) flatten_body(S, p);
    __syncthreads();
    const uint32_t comps = block_compact(FirstComponents{S}, n);
    if (threadIdx.x == 0) {
        S.stat[kStEdges] = edges;
        S.stat[kStComps] = comps;
    }
    if (comps > 1) block_nodes_and_seeds(S, 0);
}
// After a round's search: the merge, and the nodes and seeds of the next.
__global__ void __launch_bounds__(kSmallThreads) small_round_kernel(BorState S) {
    const int64_t ncomp = S.stat[kStComps];
    if (ncomp <= 1) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t r = S.stat[kStRounds]++;
        if (r < kMaxRounds) S.stat[kStHistory + r] = (uint32_t)ncomp;
    }
    for (int64_t p = threadIdx.x; p < S.n; p += blockDim.x) stage_b_body(S, p);
    __syncthreads();
    for (int64_t p = threadIdx.x; p < S.n; p += blockDim.x) stage_c_body(S, p);
    __syncthreads();
    for (int64_t i = threadIdx.x; i < ncomp; i += blockDim.x) select_body(S, i);
    __syncthreads();
    block_merge(S, ncomp);
    if (S.stat[kStComps] > 1) block_nodes_and_seeds(S, 1);
}

// ------------------------------------------- reference tie mode, per round
// The reference's choice of a component's edge (boruvka.py:34-60 over the
// candidates of boruvka.py:290-331, its loops run in order): the point of
// lowest caller index among those attaining the component's least weight w,
// and that point's first candidate at weight w in its KD-tree walk.  (The
// shared bound never cuts that point's search short: when it runs, the bound
// only holds weights above w.)  With the component keys packed as (weight,
// caller index of the choosing point), the key's low word is that point.
__global__ void ref_winner_kernel(const int32_t* __restrict__ reps, int64_t nrep,
                                  const unsigned long long* __restrict__ keyA,
                                  const int32_t* __restrict__ rank, int32_t* __restrict__ winner) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrep) return;
    const int32_t c = reps[i];
    const unsigned long long key = keyA[c];
    winner[c] = key == ~0ull ? -1 : rank[(uint32_t)(key & 0xffffffffu)];
}

// One warp per component: every point of another component at exactly the
// winner's weight w (max(rdist, core, core) == w, the search's expression)
// is found by a walk of the bucket tree limited to nodes that can hold one;
// the reference's walk meets them in its own tree's depth-first order, and
// the first of them in that order (ref_before) is the edge's far end.
template <int DIM, int SP>
__global__ void __launch_bounds__(kSW * 32) tie_walk_kernel(
    IndexView ix, RefTreeView rt, const int32_t* __restrict__ reps, int64_t nrep,
    const int32_t* __restrict__ comp, const float* __restrict__ core2,
    const int2* __restrict__ nc, const int32_t* __restrict__ winner,
    const float* __restrict__ cand_w, int32_t* __restrict__ cand_q, int32_t* __restrict__ tgt,
    int* __restrict__ missing) {
    __shared__ int32_t s_stack[kSW][kStack];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * kSW + warp;
    if (i >= nrep) return;
    const int32_t c = reps[i];
    const int32_t p = winner[c];
    if (p < 0) {
        if (lane == 0) {
            tgt[c] = -1;
            atomicOr(missing, 1);
        }
        return;
    }
    const float w = cand_w[p], cp = core2[p];
    float q[DIM];
    {
        float t[SP];
        load_pt<SP>(ix.pts, p, t);
#pragma unroll
        for (int j = 0; j < DIM; ++j) q[j] = t[j];
    }
    int32_t best = -1;
    int64_t best_pos = -1;
    int32_t* st = s_stack[warp];
    const int64_t first_leaf = ix.slots - 1;
    auto wanted = [&](int64_t node) {
        const int2 ncn = nc[node];
        if (ncn.x == c || ncn.x == kEmpty || __int_as_float(ncn.y) > w) return false;
        float b[2 * SP];
        load_box<SP>(ix.box, node, b);
        return box_lb_n<DIM, SP>(b, q) <= w;
    };
    int sp = 0;
    if (wanted(0)) {
        if (lane == 0) st[0] = 0;
        sp = 1;
    }
    __syncwarp();
    while (sp > 0) {
        --sp;
        const int32_t node = st[sp];
        __syncwarp();
        if (node >= first_leaf) {
            const int64_t leaf = node - first_leaf;
            const int64_t qp = leaf * kLeaf + lane;
            int32_t my = -1;
            int64_t mypos = -1;
            if (leaf < ix.nleaves && qp < ix.n && comp[qp] != c) {
                const float ck = core2[qp];
                if (!(ck > w)) {
                    float x[SP];
                    load_pt<SP>(ix.pts, qp, x);
                    const float wt = fmaxf(fmaxf(rdist_rn<DIM>(q, x), cp), ck);
                    if (wt == w) {
                        my = (int32_t)qp;
                        mypos = rt.pos[ix.orig[qp]];
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int32_t other = __shfl_xor_sync(kFull, my, o);
                const int64_t opos = __shfl_xor_sync(kFull, mypos, o);
                if (other >= 0 && (my < 0 || ref_before(rt, q, opos, mypos))) {
                    my = other;
                    mypos = opos;
                }
            }
            if (my >= 0 && (best < 0 || ref_before(rt, q, mypos, best_pos))) {
                best = my;
                best_pos = mypos;
            }
            continue;
        }
        const int32_t l = 2 * node + 1, r = l + 1;
        const bool wl = wanted(l), wr = wanted(r);
        if (lane == 0) {
            int t = sp;
            if (wl) st[t++] = l;
            if (wr) st[t] = r;
        }
        sp += (wl ? 1 : 0) + (wr ? 1 : 0);
        __syncwarp();
    }
    if (lane == 0) {
        if (best < 0) {
            tgt[c] = -1;
            atomicOr(missing, 2);
        } else {
            cand_q[p] = best;
            tgt[c] = comp[best];
        }
    }
}

// The reference adds the components' edges in its dict order (each
// component's lowest caller index, cmin) and skips an edge whose ends are
// already joined.  The edges form a functional graph on components; an edge
// is skipped exactly when it closes its part's cycle, i.e. it is the cycle's
// edge of largest cmin.  Pointer doubling finds every cycle's largest cmin.
__global__ void crep_init_kernel(const int32_t* __restrict__ reps, int64_t nrep,
                                 const int32_t* __restrict__ tgt, const int32_t* __restrict__ cmin,
                                 int32_t* __restrict__ nxt, int32_t* __restrict__ mx) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrep) return;
    const int32_t c = reps[i];
    nxt[c] = tgt[c] >= 0 ? tgt[c] : c;
    mx[c] = cmin[c];
}
__global__ void crep_step_kernel(const int32_t* __restrict__ reps, int64_t nrep,
                                 const int32_t* __restrict__ nxt, const int32_t* __restrict__ mx,
                                 int32_t* __restrict__ nxt2, int32_t* __restrict__ mx2,
                                 int* __restrict__ changed) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrep) return;
    const int32_t c = reps[i], x = nxt[c];
    nxt2[c] = nxt[x];
    const int32_t a = mx[c], b = mx[x];
    mx2[c] = max(a, b);
    if (changed && b > a) *changed = 1;
}
__global__ void crep_drop_kernel(const int32_t* __restrict__ reps, int64_t nrep,
                                 const int32_t* __restrict__ nxt, const int32_t* __restrict__ mx,
                                 const int32_t* __restrict__ cmin, int32_t* __restrict__ tgt) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrep) return;
    const int32_t c = reps[i];
    if (tgt[c] >= 0 && mx[nxt[c]] == cmin[c]) tgt[c] = -1;
}
__global__ void finalize_edges_kernel(int64_t m, const int32_t* __restrict__ src,
                                      const int32_t* __restrict__ dst,
                                      const float* __restrict__ w2, double* __restrict__ edges) {
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m) return;
    edges[3 * e + 0] = (double)src[e];
    edges[3 * e + 1] = (double)dst[e];
    edges[3 * e + 2] = __dsqrt_rn((double)w2[e]);
}

// Warps per bucket (or per 32 listed points), as for the kNN: with few of
// them the latency of one walk is the search's time.  Listed points, each
// walking from the root, have the least to share and take twice as many.  (All
// searches, ms with 20 / 40 / 80 / 160 warps wanted per SM: 60k x 13-D 3.85 / 3.59
// / 4.36 / 6.07, 20k x 2-D 0.142 / 0.131 / 0.139 / 0.162; the lists alone, 40 / 80 /
// 160: 200k x 4-D 1.35 / 1.24 / 1.33, 20k x 2-D 0.130 / 0.126 / 0.129.)
constexpr int64_t kSearchWarpsWanted = 40 * 152;
int search_split(int64_t groups, int64_t wanted) {
    int split = 1;
    while (split < 32 && 2 * split * groups <= wanted) split *= 2;
    return split;
}

template <int DIM>
int launch_search(Workspace& ws, const fhg_index& ix, const int8_t* knn_open, const BorState& S,
                  bool one_pass, bool* try_sparse) {
    constexpr int SP = DIM <= 4 ? 4 : (DIM <= 8 ? 8 : DIM);  // as in the kNN kernel
    const int64_t n = ix.n;
    cudaStream_t s = ws.stream();
    auto run = [&](int pass, const int32_t* list, int64_t len) -> int {
        const int64_t groups = list ? (len + 31) / 32 : ix.nleaves;
        const int split = search_split(groups, list ? 2 * kSearchWarpsWanted : kSearchWarpsWanted);
        Stage stage(s, "search_kernel");
        ::fhg::note_launch();
        search_kernel<DIM, SP><<<grid_for(groups * split, kSW), kSW * 32, 0, s>>>(
            view_of(ix), knn_open, S.core2, S.comp, S.nc, S.keyA, S.cand_w, S.cand_q, pass, list,
            len, S.ref_ties, split, S.stat);
        FHG_CUDA(cudaGetLastError());
        return FHG_OK;
    };
    // When few points search (early rounds: most points' best edge is settled
    // by the seeds), one pass runs on a list of them, 32 to a warp, each from
    // the root -- instead of a warp per bucket walking for one or two of its
    // lanes.  Searching only grows with the components, so after the first
    // dense round the list is not made again.
    if (*try_sparse) {
        Workspace tmp(ws);
        uint32_t* cnt;
        int32_t* list;
        FHG_TRY(tmp.alloc(&list, (size_t)n));
        FHG_TRY(tmp.alloc(&cnt, 1));
        FHG_TRY(compact(tmp, SearchingPoints{S, knn_open, list}, n, cnt));
        uint32_t h_cnt = 0;
        FHG_CUDA(cudaMemcpyAsync(&h_cnt, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        FHG_CUDA(cudaStreamSynchronize(s));
        const int64_t ns = h_cnt;
        if (ns == 0) return FHG_OK;
        *try_sparse = ns * kSparseDen < n * kSparseNum;
        if (*try_sparse) return run(2, list, ns);
    }
    if (one_pass || ix.slots <= 32) return run(2, nullptr, 0);
    FHG_TRY(run(0, nullptr, 0));
    return run(1, nullptr, 0);
}

template <int DIM>
int launch_tie_walk(const fhg_index& ix, const RefTree& rt, const int32_t* reps, int64_t nrep,
                    const int32_t* comp, const float* core2, const int2* nc,
                    const int32_t* winner, const float* cand_w, int32_t* cand_q, int32_t* tgt,
                    int* missing, cudaStream_t s) {
    constexpr int SP = DIM <= 4 ? 4 : (DIM <= 8 ? 8 : DIM);
    if (nrep <= 0) return FHG_OK;
    Stage stage(s, "tie_walk_kernel");
    ::fhg::note_launch();
    tie_walk_kernel<DIM, SP><<<grid_for(nrep, kSW), kSW * 32, 0, s>>>(
        view_of(ix), view_of(rt), reps, nrep, comp, core2, nc, winner, cand_w, cand_q, tgt,
        missing);
    FHG_CUDA(cudaGetLastError());
    return FHG_OK;
}

int tie_walk(const fhg_index& ix, const RefTree& rt, const int32_t* reps, int64_t nrep,
             const int32_t* comp, const float* core2, const int2* nc, const int32_t* winner,
             const float* cand_w, int32_t* cand_q, int32_t* tgt, int* missing, cudaStream_t s) {
#define FHG_TW(D) launch_tie_walk<D>(ix, rt, reps, nrep, comp, core2, nc, winner, cand_w, cand_q, \
                                     tgt, missing, s)
    switch (ix.d) {
        case 1: return FHG_TW(1);
        case 2: return FHG_TW(2);
        case 3: return FHG_TW(3);
        case 4: return FHG_TW(4);
        case 5: return FHG_TW(5);
        case 6: return FHG_TW(6);
        case 7: return FHG_TW(7);
        case 8: return FHG_TW(8);
        default:
            if (ix.d <= 16) return FHG_TW(16);
            return FHG_TW(32);
    }
#undef FHG_TW
}

int search_round(Workspace& ws, const fhg_index& ix, const int8_t* knn_open, const BorState& S,
                 bool one_pass, bool* try_sparse) {
    switch (ix.d) {
        case 1: return launch_search<1>(ws, ix, knn_open, S, one_pass, try_sparse);
        case 2: return launch_search<2>(ws, ix, knn_open, S, one_pass, try_sparse);
        case 3: return launch_search<3>(ws, ix, knn_open, S, one_pass, try_sparse);
        case 4: return launch_search<4>(ws, ix, knn_open, S, one_pass, try_sparse);
        case 5: return launch_search<5>(ws, ix, knn_open, S, one_pass, try_sparse);
        case 6: return launch_search<6>(ws, ix, knn_open, S, one_pass, try_sparse);
        case 7: return launch_search<7>(ws, ix, knn_open, S, one_pass, try_sparse);
        case 8: return launch_search<8>(ws, ix, knn_open, S, one_pass, try_sparse);
        default:
            if (ix.d <= 16) return launch_search<16>(ws, ix, knn_open, S, one_pass, try_sparse);
            return launch_search<32>(ws, ix, knn_open, S, one_pass, try_sparse);
    }
}

#define LAUNCH(kernel, count, ...)                                                   \
    do {                                                                             \
        if ((count) > 0) {                                                           \
            ::fhg::note_launch(); \
            kernel<<<grid_for((count), 256), 256, 0, s>>>(__VA_ARGS__);              \
            FHG_CUDA(cudaGetLastError());                                            \
        }                                                                            \
    } while (0)

}  // namespace

// The tie rule of the calling host thread (fhg_set_tie_rule).
namespace {
thread_local int t_tie_rule = FHG_TIES_CANONICAL;
}
int tie_rule() { return t_tie_rule; }
int set_tie_rule(int rule) {
    const int old = t_tie_rule;
    t_tie_rule = rule;
    return old;
}

int finalize_edges(const MstResult& r, double* edges, cudaStream_t s) {
    LAUNCH(finalize_edges_kernel, r.m, r.m, r.src, r.dst, r.w2, edges);
    return FHG_OK;
}

int boruvka_mst(Workspace& ws, const fhg_index& ix, int min_samples, MstResult* out,
                float* core_o, int32_t* nbr_o, const float* weights, int weighted_k,
                bool any_order) {
    cudaStream_t s = ws.stream();
    const int64_t n = ix.n;
    const bool weighted = weights != nullptr && n > 1;
    const int ref_ties = tie_rule() == FHG_TIES_REFERENCE ? 1 : 0;
    // the reference's k (boruvka.py:561-585)
    const int kq = weighted ? weighted_k : (min_samples > 1 ? min_samples + 1 : 2);
    const int k = (int)(kq < n ? kq : n);  // neighbours that exist
    *out = MstResult();
    if (kq < 1) {
        set_error("weighted kNN: k = %d (2 * min_samples / mean weight) is below 1", kq);
        return FHG_ERR_INVALID;
    }
    // lists of up to 64 live in registers (and the reference tie mode's
    // re-query takes no more); longer ones in shared memory
    const int k_max = ref_ties ? 64 : kKnnMaxK;
    if (k > k_max) {
        if (weighted)
            set_error("weighted kNN: k = %d (2 * min_samples / mean weight) exceeds %d%s", kq,
                      k_max, ref_ties ? " in the reference tie mode" : "");
        else
            set_error("min_samples must be at most %d (got %d)%s", k_max - 1, min_samples,
                      ref_ties ? " in the reference tie mode" : "");
        return FHG_ERR_UNSUPPORTED;
    }
    const int64_t m_cap = n > 1 ? n - 1 : 1;
    FHG_TRY(ws.alloc(&out->src, (size_t)m_cap));
    FHG_TRY(ws.alloc(&out->dst, (size_t)m_cap));
    FHG_TRY(ws.alloc(&out->w2, (size_t)m_cap));

    float *knn_d, *core2;
    int32_t* knn_s;
    FHG_TRY(ws.alloc(&knn_d, (size_t)(n * k)));
    FHG_TRY(ws.alloc(&knn_s, (size_t)(n * k)));
    int8_t* knn_open;  // the kNN kernel's tie flags, then "seed not provably final"
    FHG_TRY(ws.alloc(&knn_open, (size_t)n));
    // the neighbours[:, 1:] matrix (kq - 1 columns) straight from the kNN kernel
    const RadiusUse* ru = k <= 64 ? radius_in_use() : nullptr;  // (radius passes: k <= 64)
    if (ru)
        FHG_TRY(knn_with_radius(ix, k, *ru, knn_d, knn_s, nullptr, nbr_o, s, knn_open, kq - 1, 1));
    else
        FHG_TRY(index_knn(ix, k, knn_d, knn_s, nullptr, nbr_o, s, knn_open, kq - 1, 1));
    // the reference tie mode breaks ties in the order of the reference's own
    // KD-tree, built here exactly; its kNN lists (and so round 0 and the
    // neighbour matrix) list equal distances in the order of the reference's
    // query and heap, and replace the engine's rows (the same distances)
    RefTree rt;
    if (ref_ties && n > 1) {
        FHG_TRY(ref_tree_build(ws, ix, &rt));
        FHG_TRY(ref_knn(rt, ix, kq, weighted, knn_open, knn_d, knn_s, nbr_o, kq - 1, s));
    }
    FHG_TRY(ws.alloc(&core2, (size_t)n));
    if (weighted) {
        float* w_s;
        float w_last = 0.0f;
        FHG_TRY(ws.alloc(&w_s, (size_t)n));
        LAUNCH(gather_weights_kernel, n, n, ix.orig, weights, w_s);
        FHG_CUDA(cudaMemcpyAsync(&w_last, weights + (n - 1), sizeof(float), cudaMemcpyDeviceToHost,
                                 s));
        FHG_CUDA(cudaStreamSynchronize(s));
        LAUNCH(weighted_core_kernel, n, n, k, kq, min_samples, knn_d, knn_s, w_s, w_last, core2,
               knn_open);
    }
    const int core_from_knn = weighted ? 0 : 1;
    const bool small = n > 1 && !ref_ties && n <= kSmallPoints && n * k <= kSmallEntries;
    if (!small && (core_from_knn || core_o || nbr_o))
        LAUNCH(core_outputs_kernel, n, n, k, kq, min_samples, core_from_knn, knn_d, core2,
               knn_open, ix.orig, core_o, nbr_o);
    if (n < 2) return FHG_OK;

    BorState S;
    S.n = n;
    S.nleaves = ix.nleaves;
    S.slots = ix.slots;
    S.k = k;
    S.ref_ties = ref_ties;
    S.plain_d = weighted ? 1 : 0;
    S.orig = ix.orig;
    S.rank = ix.rank;
    S.knn_d = knn_d;
    S.knn_s = knn_s;
    S.core2 = core2;
    S.src = out->src;
    S.dst = out->dst;
    S.w2 = out->w2;
    for (int32_t** p : {&S.target, &S.par, &S.comp, &S.cmin, &S.reps, &S.rep_cmin, &S.next_reps,
                        &S.next_cmin, &S.winner, &S.tgt, &S.cand_q})
        FHG_TRY(ws.alloc(p, (size_t)n));
    FHG_TRY(ws.alloc(&S.w0, (size_t)n));
    FHG_TRY(ws.alloc(&S.keyA, (size_t)n));
    FHG_TRY(ws.alloc(&S.keyB, (size_t)n));
    FHG_TRY(ws.alloc(&S.cand_w, (size_t)n));
    FHG_TRY(ws.alloc(&S.exhausted, (size_t)n));
    FHG_TRY(ws.alloc(&S.nc, (size_t)ix.nnodes));
    FHG_TRY(ws.alloc(&S.stat, (size_t)kStWords));
    uint32_t st[kStWords];
    auto read_stat = [&]() -> int {
        FHG_CUDA(cudaMemcpyAsync(st, S.stat, sizeof st, cudaMemcpyDeviceToHost, s));
        FHG_CUDA(cudaStreamSynchronize(s));
        return FHG_OK;
    };
    // the pointer-doubling buffers of round 0 (points) and of the reference
    // tie mode's rounds (components)
    int32_t *nxt, *mx, *nxt2, *mx2;
    for (int32_t** p : {&nxt, &mx, &nxt2, &mx2}) FHG_TRY(ws.alloc(p, (size_t)n));
    // round-0 edges by caller index of the choosing point (the reference's
    // order), or by index position when the order does not matter
    const int by_caller = any_order ? 0 : 1;

    // ---- round 0: kNN-seeded links (boruvka.py:474)
    {
        Stage stage(s, "boruvka_round0");
        if (small) {
            ::fhg::note_launch();
            small_round0_kernel<<<1, kSmallThreads, 0, s>>>(S, kq, min_samples, core_from_knn,
                                                            knn_open, core_o, nbr_o, by_caller, nxt,
                                                            mx, nxt2, mx2);
            FHG_CUDA(cudaGetLastError());
        } else {
            FHG_CUDA(cudaMemsetAsync(S.stat, 0, sizeof st, s));
            LAUNCH(round0_kernel, n, S);
            FHG_TRY(read_stat());
            if (st[kStEqual]) {
                LAUNCH(cyc_init_kernel, n, S, nxt, mx);
                // link chains are short: every fourth step reports whether it
                // changed anything, and the doubling stops at the first that
                // did not
                int* grew = reinterpret_cast<int*>(S.stat + kStEqual);
                const int R = bits_for(n) + 1;
                for (int r = 0; r < R; ++r) {
                    const bool check = (r & 3) == 3 && r + 1 < R;
                    if (check) FHG_CUDA(cudaMemsetAsync(grew, 0, sizeof(int), s));
                    LAUNCH(cyc_step_kernel, n, n, nxt, mx, nxt2, mx2, check ? grew : nullptr);
                    std::swap(nxt, nxt2);
                    std::swap(mx, mx2);
                    if (check) {
                        FHG_TRY(read_stat());
                        if (!st[kStEqual]) break;
                    }
                }
                LAUNCH(cyc_drop_kernel, n, S, nxt, mx);
            }
            FHG_TRY(compact(ws, Round0Edges{S, by_caller}, n, S.stat + kStEdges));
            LAUNCH(union_targets_kernel, n, S);
            LAUNCH(flatten_kernel, n, S);
            FHG_TRY(compact(ws, FirstComponents{S}, n, S.stat + kStComps));
        }
    }

    int rounds = 0;
    bool dense = false;  // small inputs never make a list of the searching points
    bool try_sparse = true;  // until a round's global pass is dense
    if (small) {
        // two rounds between the host's reads: a round after the last costs
        // less than a read
        for (;;) {
            FHG_TRY(read_stat());
            if (st[kStComps] <= 1 || st[kStMissing] || st[kStRounds] >= kMaxRounds) break;
            for (int r = 0; r < 2; ++r) {
                {
                    Stage stage(s, "boruvka_search");
                    FHG_TRY(search_round(ws, ix, knn_open, S, /*one_pass=*/true, &dense));
                }
                Stage stage(s, "boruvka_merge");
                ::fhg::note_launch();
                small_round_kernel<<<1, kSmallThreads, 0, s>>>(S);
                FHG_CUDA(cudaGetLastError());
            }
        }
        rounds = (int)st[kStRounds];
        for (int r = 0; r < rounds && r < kMaxRounds; ++r)  // C_r of the rounds
            profile_count("boruvka_components", (double)st[kStHistory + r]);
    } else {
        FHG_TRY(read_stat());
        while (st[kStComps] > 1) {
            const int64_t ncomp = st[kStComps], edges = st[kStEdges];
            if (rounds >= kMaxRounds) break;
            profile_count("boruvka_components", (double)ncomp);  // C_r of the round
            {  // node_comp (boruvka.py:98-124), bottom-up
                Stage stage(s, "boruvka_nodes");
                int64_t width = (ix.slots + kNodeLeaves - 1) / kNodeLeaves;
                ::fhg::note_launch();
                node_chunk_kernel<<<(unsigned)width, kNodeThreads, 0, s>>>(S, rounds > 0 ? 1 : 0);
                FHG_CUDA(cudaGetLastError());
                while (width > 1) {
                    const int64_t blocks = (width + kNodeTop - 1) / kNodeTop;
                    ::fhg::note_launch();
                    node_top_kernel<<<(unsigned)blocks, kNodeTop / 2, 0, s>>>(S.nc, width);
                    FHG_CUDA(cudaGetLastError());
                    width = blocks;
                }
            }
            {
                Stage stage(s, "boruvka_search");
                LAUNCH(seed_kernel, n, S);
                FHG_TRY(search_round(ws, ix, knn_open, S, /*one_pass=*/false, &try_sparse));
            }
            Stage merge_stage(s, "boruvka_merge");
            if (ref_ties) {
                LAUNCH(ref_winner_kernel, ncomp, S.reps, ncomp, S.keyA, ix.rank, S.winner);
                FHG_TRY(tie_walk(ix, rt, S.reps, ncomp, S.comp, core2, S.nc, S.winner, S.cand_w,
                                 S.cand_q, S.tgt, reinterpret_cast<int*>(S.stat + kStMissing), s));
                LAUNCH(crep_init_kernel, ncomp, S.reps, ncomp, S.tgt, S.cmin, nxt, mx);
                int* grew = reinterpret_cast<int*>(S.stat + kStEqual);
                const int R = bits_for(ncomp) + 1;
                for (int r = 0; r < R; ++r) {
                    const bool check = (r & 3) == 3 && r + 1 < R;
                    if (check) FHG_CUDA(cudaMemsetAsync(grew, 0, sizeof(int), s));
                    LAUNCH(crep_step_kernel, ncomp, S.reps, ncomp, nxt, mx, nxt2, mx2,
                           check ? grew : nullptr);
                    std::swap(nxt, nxt2);
                    std::swap(mx, mx2);
                    if (check) {
                        FHG_TRY(read_stat());
                        if (!st[kStEqual]) break;
                    }
                }
                LAUNCH(crep_drop_kernel, ncomp, S.reps, ncomp, nxt, mx, S.cmin, S.tgt);
            } else {
                LAUNCH(stage_b_kernel, n, S);
                LAUNCH(stage_c_kernel, n, S);
            }
            if (ncomp <= kBlockMerge) {
                ::fhg::note_launch();
                merge_kernel<<<1, kSmallThreads, 0, s>>>(S, ncomp);
                FHG_CUDA(cudaGetLastError());
            } else {
                if (!ref_ties) LAUNCH(select_kernel, ncomp, S, ncomp);
                FHG_TRY(compact(ws, RoundEdges{S}, ncomp, S.stat + kStAdded));
                LAUNCH(merge_cmin_kernel, ncomp, S, ncomp);
                FHG_TRY(compact(ws, MergedComponents{S}, ncomp, S.stat + kStComps));
                std::swap(S.reps, S.next_reps);
                std::swap(S.rep_cmin, S.next_cmin);
            }
            FHG_TRY(read_stat());
            if (st[kStMissing] || st[kStEdges] - edges != ncomp - st[kStComps]) {
                set_error("boruvka round %d: inconsistent merge (added %lld, components %lld -> "
                          "%lld, missing=%d)", rounds, (long long)(st[kStEdges] - edges),
                          (long long)ncomp, (long long)st[kStComps], (int)st[kStMissing]);
                return FHG_ERR_NO_CONVERGENCE;
            }
            ++rounds;
        }
    }
    if (st[kStComps] > 1 || st[kStMissing] || (int64_t)st[kStEdges] + st[kStComps] != n) {
        set_error("boruvka: no convergence after %d rounds (%lld components, %lld edges left, "
                  "missing=%d)", rounds, (long long)st[kStComps],
                  (long long)(n - 1 - (int64_t)st[kStEdges]), (int)st[kStMissing]);
        return FHG_ERR_NO_CONVERGENCE;
    }
    out->m = st[kStEdges];
    out->rounds = rounds;
    return FHG_OK;
}

}  // namespace fhg
