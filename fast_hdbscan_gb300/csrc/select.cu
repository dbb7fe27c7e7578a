// Cluster selection, labels and membership strengths over the condensed tree.
//
//   stabilities   cluster_trees.py:656 score_condensed_tree_nodes -- float32,
//                 accumulated in row order.  Rows are stably sorted by parent,
//                 then each cluster sums its own rows in order, so every
//                 rounding step matches the reference.
//   EOM           cluster_trees.py:694 eom_recursion / :724
//                 extract_eom_clusters -- evaluated bottom-up over the (small)
//                 cluster tree, one depth level at a time in a single block;
//                 child totals are float64 sums in row order.
//   leaf          cluster_trees.py:369 cluster_tree_leaves.
//   labels        cluster_trees.py:944 get_cluster_label_vector -- the
//                 reference's union-find over unselected rows gives every
//                 point the nearest selected cluster above its row's parent,
//                 computed here by pointer doubling over clusters.
//   probabilities cluster_trees.py:999-1031.
#include "compact.cuh"
#include "primitives.cuh"
#include "trees.cuh"

namespace fhg {
namespace {

constexpr int kEomThreads = 1024;

// Maximum of non-negative floats as bits, with an atomic only where it grows.
__device__ __forceinline__ void max_bits(unsigned int* to, unsigned int b) {
    if (b > *(volatile unsigned int*)to) atomicMax(to, b);
}
// One pass over the rows: the row of every point and cluster, the largest
// lambda under the root (root_max) and of every cluster's points (death), and
// -- with key -- the parent keys and the row numbers to be sorted by them.
// A few clusters have most rows, and what bounds this is how many warps turn to
// the same words: a block brings the maxima of its rows together first, in a
// small table by cluster (rows of a cluster stand together; a cluster whose
// place is taken goes to its word directly), and takes them on once (10M rows:
// 1.48 -> 0.83 ms, 1M: 98 -> 54 us, with a maximum per warp before).
constexpr int kFactsThreads = 256, kFactsRows = 4, kFactsSlots = 64;
__global__ void __launch_bounds__(kFactsThreads) row_facts_kernel(
    int64_t rows, int64_t n, const int32_t* __restrict__ parent,
    const int32_t* __restrict__ child, const float* __restrict__ lam,
    const float* __restrict__ csize, int32_t* __restrict__ row_of_point,
    int32_t* __restrict__ row_of_cluster, unsigned int* root_max, unsigned int* death,
    uint32_t* __restrict__ key, int32_t* __restrict__ order) {
    __shared__ int32_t s_cluster[kFactsSlots];
    __shared__ unsigned int s_max[kFactsSlots], s_root;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < kFactsSlots) {
        s_cluster[threadIdx.x] = -1;
        s_max[threadIdx.x] = 0u;
    }
    if (threadIdx.x == 0) s_root = 0u;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * (kFactsThreads * kFactsRows) + threadIdx.x;
#pragma unroll
    for (int t = 0; t < kFactsRows; ++t) {
        const int64_t r = base + t * kFactsThreads;
        const bool here = r < rows;
        int32_t c = -1;
        unsigned int b = 0u;  // (non-negative floats order like their bits)
        bool pt = false;
        if (here) {
            c = parent[r] - (int32_t)n;
            b = __float_as_uint(lam[r]);
            pt = csize[r] == 1.0f;
            const int32_t x = child[r];
            if (x >= n) row_of_cluster[x - n] = (int32_t)r;
            else row_of_point[x] = (int32_t)r;
            if (key) {
                key[r] = (uint32_t)c;
                order[r] = (int32_t)r;
            }
        }
        const unsigned top = __reduce_max_sync(kFull, c == 0 ? b : 0u);
        if (lane == 0 && top) atomicMax(&s_root, top);
        const unsigned pts = __ballot_sync(kFull, pt);
        if (pt) {
            const unsigned peers = __match_any_sync(pts, c);
            const unsigned m = __reduce_max_sync(peers, b);
            if (lane == __ffs(peers) - 1) {
                const int slot = c & (kFactsSlots - 1);
                const int32_t was = atomicCAS(&s_cluster[slot], -1, c);
                if (was == -1 || was == c) atomicMax(&s_max[slot], m);
                else max_bits(&death[c], m);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < kFactsSlots && s_cluster[threadIdx.x] >= 0)
        max_bits(&death[s_cluster[threadIdx.x]], s_max[threadIdx.x]);
    if (threadIdx.x == 0 && s_root) max_bits(root_max, s_root);
}
// lambda * size of every row, in parent-grouped row order (contiguous per
// cluster), so that each cluster's sequential sum below streams its addends.
// The sorted keys' runs are the clusters' ranges [start, start + cnt).
__global__ void products_kernel(int64_t rows, const uint32_t* __restrict__ key,
                                const int32_t* __restrict__ order,
                                const float* __restrict__ lam, const float* __restrict__ csize,
                                float* __restrict__ prod, int64_t* __restrict__ start,
                                int64_t* __restrict__ end) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= rows) return;
    int32_t r = order[j];
    prod[j] = __fmul_rn(lam[r], csize[r]);
    const uint32_t c = key[j];
    if (j == 0 || key[j - 1] != c) start[c] = j;
    if (j + 1 == rows || key[j + 1] != c) end[c] = j + 1;
}
// The float32 sum of a cluster's products, strictly in row order (a float32 sum
// is not associative, so the order is the result): one warp per cluster.  The
// lanes read 32 products together, the next ones while these are added, and all
// add the same chain; a thread per cluster waited for each of its loads (1M
// points, min_cluster_size 500: 218 -> 29 us).  Clusters of kBigRows rows or
// more are summed by score_big_kernel.  Above kScoreWarps clusters a warp takes
// 32 of them, a lane each where they have up to kLaneRows rows: most are small
// then, and a warp for each leaves its lanes idle (1M clusters of 10 rows on
// average: 286 -> 24 us).
constexpr int32_t kBigRows = 2048;
__device__ __forceinline__ float score_start(int64_t c, const int32_t* __restrict__ row_of_cluster,
                                             const float* __restrict__ lam,
                                             const float* __restrict__ csize) {
    float s = 0.0f;
    if (c > 0) {
        int32_t r = row_of_cluster[c];
        if (r >= 0 && csize[r] > 1.0f) s = __fmul_rn(-lam[r], csize[r]);
    }
    return s;
}
// s + v[0] + v[1] + ... + v[len - 1] by one warp.
__device__ __forceinline__ float warp_sum(float s, const float* __restrict__ p, int len) {
    const int lane = threadIdx.x & 31;
    float v = lane < len ? __ldg(p + lane) : 0.0f;
    for (int j = 0; j < len; j += 32) {
        const float next = j + 32 + lane < len ? __ldg(p + j + 32 + lane) : 0.0f;
        if (len - j >= 32) {
#pragma unroll
            for (int u = 0; u < 32; ++u) s = __fadd_rn(s, __shfl_sync(kFull, v, u));
        } else {
            for (int u = 0; u < len - j; ++u) s = __fadd_rn(s, __shfl_sync(kFull, v, u));
        }
        v = next;
    }
    return s;
}
__global__ void score_kernel(int64_t C, const int64_t* __restrict__ start,
                             const int64_t* __restrict__ end, const float* __restrict__ prod,
                             const int32_t* __restrict__ row_of_cluster,
                             const float* __restrict__ lam, const float* __restrict__ csize,
                             float* __restrict__ score) {
    const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= C) return;
    const int64_t b = start[c];
    const int len = (int)min(end[c] - b, (int64_t)kBigRows);
    if (len >= kBigRows) return;
    const float s = warp_sum(score_start(c, row_of_cluster, lam, csize), prod + b, len);
    if ((threadIdx.x & 31) == 0) score[c] = s;
}
constexpr int64_t kScoreWarps = 16384;
constexpr int kLaneRows = 64;
__global__ void score_many_kernel(int64_t C, const int64_t* __restrict__ start,
                                  const int64_t* __restrict__ end, const float* __restrict__ prod,
                                  const int32_t* __restrict__ row_of_cluster,
                                  const float* __restrict__ lam, const float* __restrict__ csize,
                                  float* __restrict__ score) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int64_t b = 0;
    int len = kBigRows;  // (past the clusters: nothing to do)
    float s = 0.0f;
    if (c < C) {
        b = start[c];
        len = (int)min(end[c] - b, (int64_t)kBigRows);
        s = score_start(c, row_of_cluster, lam, csize);
        if (len <= kLaneRows) {
            int j = 0;
            for (; j + 8 <= len; j += 8) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = __ldg(prod + b + j + u);
#pragma unroll
                for (int u = 0; u < 8; ++u) s = __fadd_rn(s, v[u]);
            }
            for (; j < len; ++j) s = __fadd_rn(s, __ldg(prod + b + j));
            score[c] = s;
        }
    }
    for (unsigned m = __ballot_sync(kFull, len > kLaneRows && len < kBigRows); m; m &= m - 1u) {
        const int i = __ffs(m) - 1;
        const float t = warp_sum(__shfl_sync(kFull, s, i), prod + __shfl_sync(kFull, b, i),
                                 __shfl_sync(kFull, len, i));
        if (lane == i) score[c] = t;
    }
}
// One block per cluster of kBigRows rows or more: the same sequential sum by
// one thread, fed from shared memory -- the other warps stage the next chunk
// of products while the current one is summed, so that the chain of
// dependent additions never waits for memory.
constexpr int kScoreThreads = 256;
constexpr int kScoreChunk = 4096;
// The first bit set from i on, or kScoreThreads.
__device__ __forceinline__ int next_large(const unsigned* bits, int i) {
    for (; i < kScoreThreads; i = (i | 31) + 1) {
        const unsigned m = bits[i >> 5] >> (i & 31);
        if (m) return i + __ffs(m) - 1;
    }
    return kScoreThreads;
}
__global__ void __launch_bounds__(kScoreThreads) score_big_kernel(
    int64_t C, const int64_t* __restrict__ start, const int64_t* __restrict__ end,
    const float* __restrict__ prod, const int32_t* __restrict__ row_of_cluster,
    const float* __restrict__ lam, const float* __restrict__ csize, float* __restrict__ score) {
    __shared__ float buf[2][kScoreChunk];
    __shared__ unsigned s_large[kScoreThreads / 32];
    const int64_t stride = gridDim.x;
    for (int64_t c0 = blockIdx.x; c0 < C; c0 += stride * kScoreThreads) {
        // (every stride-th cluster is this block's: a look at kScoreThreads at once)
        const int64_t mine = c0 + threadIdx.x * stride;
        const unsigned large =
            __ballot_sync(kFull, mine < C && end[mine] - start[mine] >= kBigRows);
        if ((threadIdx.x & 31) == 0) s_large[threadIdx.x >> 5] = large;
        __syncthreads();
        for (int i = next_large(s_large, 0); i < kScoreThreads; i = next_large(s_large, i + 1)) {
            const int64_t c = c0 + i * stride, b = start[c], len = end[c] - b;
            const int64_t chunks = (len + kScoreChunk - 1) / kScoreChunk;
            for (int64_t j = threadIdx.x; j < kScoreChunk && j < len; j += blockDim.x)
                buf[0][j] = __ldg(prod + b + j);
            __syncthreads();
            float s = threadIdx.x == 0 ? score_start(c, row_of_cluster, lam, csize) : 0.0f;
            for (int64_t k = 0; k < chunks; ++k) {
                const int cur = (int)(k & 1);
                const int64_t base = k * kScoreChunk;
                const int cl = (int)(len - base < kScoreChunk ? len - base : kScoreChunk);
                if (threadIdx.x >= 32) {  // warps 1.. stage chunk k + 1
                    const int64_t nb = base + kScoreChunk;
                    for (int64_t j = threadIdx.x - 32; j < kScoreChunk && nb + j < len;
                         j += blockDim.x - 32)
                        buf[cur ^ 1][j] = __ldg(prod + b + nb + j);
                } else if (threadIdx.x == 0) {
                    const float* v = buf[cur];
                    int t = 0;
                    for (; t + 8 <= cl; t += 8) {
                        float x[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) x[u] = v[t + u];
#pragma unroll
                        for (int u = 0; u < 8; ++u) s = __fadd_rn(s, x[u]);
                    }
                    for (; t < cl; ++t) s = __fadd_rn(s, v[t]);
                }
                __syncthreads();  // chunk k summed, chunk k + 1 staged
            }
            if (threadIdx.x == 0) score[c] = s;
        }
        __syncthreads();
    }
}

// Cluster rows (child_size > 1) in parent-grouped row order: corder, and every
// parent's range of it [cstart, cstart + ccnt) (cstart starts as -1 unsigned).
struct ClusterRows {
    const uint32_t* key;
    const int32_t* order;
    const float* csize;
    int32_t* corder;
    uint32_t* cstart;
    int32_t* ccnt;
    __device__ bool test(int64_t j) const { return csize[order[j]] > 1.0f; }
    __device__ void emit(int64_t j, uint32_t at) const {
        corder[at] = order[j];
        atomicMin(&cstart[key[j]], at);
        atomicAdd(&ccnt[key[j]], 1);
    }
    __device__ void each(int64_t) const {}
};

// Cluster-tree structure: parent cluster (local id) and size of each cluster.
__global__ void cluster_info_kernel(int64_t C, int64_t n, const int32_t* __restrict__ row_of_cluster,
                                    const int32_t* __restrict__ parent,
                                    const float* __restrict__ csize, int32_t* __restrict__ cpar,
                                    float* __restrict__ nsize, int8_t* __restrict__ in_tree) {
    int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    if (c == 0) {
        cpar[0] = -1;
        nsize[0] = (float)(n - 1);
        in_tree[0] = 1;
        return;
    }
    int32_t r = row_of_cluster[c];
    bool ok = r >= 0 && csize[r] > 1.0f;
    cpar[c] = ok ? parent[r] - (int32_t)n : -1;
    nsize[c] = ok ? csize[r] : 0.0f;
    in_tree[c] = ok ? 1 : 0;
}

// Exclusive scan by one block of kEomThreads (len small).
__device__ void block_scan_excl(int32_t* a, int64_t len, int32_t* tmp_total) {
    __shared__ int32_t part[kEomThreads / 32];
    const int t = threadIdx.x, lane = t & 31;
    const int64_t per = (len + blockDim.x - 1) / blockDim.x;
    const int64_t b = t * per, e = b + per < len ? b + per : len;
    int32_t s = 0;
    for (int64_t i = b; i < e; ++i) s += a[i];
    int32_t x = s;  // inclusive over the warp, then over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) part[t >> 5] = x;
    __syncthreads();
    if (t < 32) {
        int32_t y = part[t];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t z = __shfl_up_sync(kFull, y, o);
            if (lane >= o) y += z;
        }
        part[t] = y;
        if (t == 31) *tmp_total = y;
    }
    __syncthreads();
    int32_t run = (t >= 32 ? part[(t >> 5) - 1] : 0) + x - s;
    for (int64_t i = b; i < e; ++i) {
        const int32_t v = a[i];
        a[i] = run;
        run += v;
    }
    __syncthreads();
}

// Single-block EOM.  What bounds it is the latency of one level after another,
// leaves to root and back: up to kEomShared clusters, everything that the levels
// read and write is first brought into shared memory (1M points, min_cluster_size
// 500: 310 -> 136 us).  Above, the scratch arrays are C entries each (dcount C +
// 2) in global memory.
constexpr int64_t kEomShared = 4096;
constexpr size_t kEomBytes = 47;  // a cluster's, and 16 for dcount
template <bool HERE>
__global__ void __launch_bounds__(kEomThreads) eom_kernel(
    int64_t C, const int32_t* __restrict__ cpar, const float* __restrict__ nsize,
    const int8_t* __restrict__ in_tree, const float* __restrict__ score,
    const uint32_t* __restrict__ start, const int32_t* __restrict__ cnt,
    const int32_t* __restrict__ order, const int32_t* __restrict__ child, int64_t n,
    double max_cs, int allow_single,
    int32_t* depth, int32_t* depth2, int32_t* jmp, int32_t* jmp2, int32_t* dcount, int32_t* byd,
    double* ret, int8_t* chose, int8_t* blocked, int32_t* flags, int32_t* sel, int64_t* n_sel) {
    const int t = threadIdx.x;
    __shared__ int32_t s_maxd, s_total;
    extern __shared__ double s_eom[];
    int32_t *kid0 = nullptr, *kids = nullptr, *nkid = nullptr;
    float* own = nullptr;
    const int32_t* up = cpar;
    const int8_t* tree = in_tree;
    if constexpr (HERE) {
        ret = s_eom;
        int32_t* at = reinterpret_cast<int32_t*>(s_eom + C);
        depth = at;
        depth2 = at + C;
        jmp = at + 2 * C;
        jmp2 = at + 3 * C;
        kid0 = at + 4 * C;
        nkid = at + 5 * C;
        int32_t* s_up = at + 6 * C;
        own = reinterpret_cast<float*>(at + 7 * C);
        dcount = at + 8 * C;  // C + 2
        chose = reinterpret_cast<int8_t*>(at + 9 * C + 4);
        blocked = chose + C;
        int8_t* s_tree = chose + 2 * C;
        for (int64_t c = t; c < C; c += blockDim.x) {
            s_up[c] = cpar[c];
            kid0[c] = (int32_t)start[c];
            nkid[c] = cnt[c];
            s_tree[c] = in_tree[c];
            // (larger than the caller's maximum: never chosen)
            own[c] = (double)nsize[c] > max_cs ? -1.0f : fmaxf(score[c], 0.0f);
        }
        up = s_up;
        tree = s_tree;
        __syncthreads();
    }
    // depth of every cluster by pointer doubling (root = 0)
    for (int64_t c = t; c < C; c += blockDim.x) {
        const bool inner = c != 0 && tree[c];
        depth[c] = inner ? 1 : 0;
        jmp[c] = inner ? up[c] : 0;
    }
    __syncthreads();
    int rounds = 1;
    while (((int64_t)1 << rounds) < C + 1) ++rounds;
    for (int r = 0; r <= rounds; ++r) {
        for (int64_t c = t; c < C; c += blockDim.x) {
            const int32_t a = jmp[c];
            depth2[c] = depth[c] + depth[a];
            jmp2[c] = jmp[a];
        }
        __syncthreads();
        int32_t* tp = depth; depth = depth2; depth2 = tp;
        tp = jmp; jmp = jmp2; jmp2 = tp;
    }
    if (t == 0) s_maxd = 0;
    if constexpr (HERE) {  // the doubling's arrays serve again
        byd = depth2;
        kids = jmp;
        flags = jmp2;
        for (int64_t c = t; c < C; c += blockDim.x)
            for (int32_t q = 0; q < nkid[c]; ++q)
                if (kid0[c] + q < C) kids[kid0[c] + q] = (int32_t)(child[order[kid0[c] + q]] - n);
    }
    __syncthreads();
    for (int64_t c = t; c < C; c += blockDim.x) {
        depth[c] = min(depth[c], (int32_t)C);  // (rows that form a cycle)
        if (tree[c]) atomicMax(&s_maxd, depth[c]);
    }
    __syncthreads();
    const int32_t maxd = s_maxd;
    // bucket clusters by depth (counting sort)
    for (int64_t d = t; d <= maxd + 1; d += blockDim.x) dcount[d] = 0;
    __syncthreads();
    for (int64_t c = t; c < C; c += blockDim.x)
        if (tree[c]) atomicAdd(&dcount[depth[c]], 1);
    __syncthreads();
    block_scan_excl(dcount, maxd + 2, &s_total);
    for (int64_t c = t; c < C; c += blockDim.x)
        if (tree[c]) byd[atomicAdd(&dcount[depth[c]], 1)] = (int32_t)c;
    __syncthreads();
    // dcount[d] is now the end of level d; level d spans [end(d-1), end(d))
    for (int32_t d = maxd; d >= 0; --d) {
        const int32_t b = d == 0 ? 0 : dcount[d - 1], e = dcount[d];
        for (int32_t j = b + t; j < e; j += blockDim.x) {
            const int32_t c = byd[j];
            chose[c] = 0;
            if (c == 0 && !allow_single) {
                ret[c] = 0.0;
                continue;
            }
            double cur, tot = 0.0;
            bool too_big = false;
            if constexpr (HERE) {
                cur = (double)own[c];
                for (int32_t q = kid0[c]; q < kid0[c] + nkid[c]; ++q) {
                    const int64_t x = q < C ? kids[q] : child[order[q]] - n;
                    tot += x >= 0 && x < C ? ret[x] : 0.0;
                }
            } else {
                cur = (double)score[c] > 0.0 ? (double)score[c] : 0.0;
                too_big = (double)nsize[c] > max_cs;
                const uint32_t b0 = start[c], e0 = b0 + (uint32_t)cnt[c];
                for (uint32_t q = b0; q < e0; ++q) tot += ret[child[order[q]] - n];
            }
            if (tot > cur || too_big) {
                ret[c] = tot;
            } else {
                ret[c] = cur;
                chose[c] = 1;
            }
        }
        __syncthreads();
    }
    for (int32_t d = 0; d <= maxd; ++d) {
        const int32_t b = d == 0 ? 0 : dcount[d - 1], e = dcount[d];
        for (int32_t j = b + t; j < e; j += blockDim.x) {
            const int32_t c = byd[j];
            if (c == 0) {
                blocked[c] = 0;
                continue;
            }
            const int32_t p = up[c];
            blocked[c] = blocked[p] || (chose[p] && (p != 0 || allow_single));
        }
        __syncthreads();
    }
    // selected ids in label order (the reference dict's insertion order)
    for (int64_t c = t; c < C; c += blockDim.x)
        flags[c] = (tree[c] && chose[c] && !blocked[c]) ? 1 : 0;
    __syncthreads();
    block_scan_excl(flags, C, &s_total);
    for (int64_t c = t; c < C; c += blockDim.x) {
        const bool on = tree[c] && chose[c] && !blocked[c];
        if (on) sel[flags[c]] = (int32_t)(n + c);
    }
    if (t == 0) *n_sel = s_total;
}

__global__ void __launch_bounds__(kEomThreads) leaf_kernel(
    int64_t C, int64_t n, const int32_t* __restrict__ cpar, const int8_t* __restrict__ in_tree,
    int32_t* __restrict__ flags, int32_t* sel, int64_t* n_sel) {
    const int t = threadIdx.x;
    __shared__ int32_t s_max, s_total;
    if (t == 0) s_max = -1;
    for (int64_t c = t; c < C; c += blockDim.x) flags[c] = 1;
    __syncthreads();
    for (int64_t c = t; c < C; c += blockDim.x)
        if (in_tree[c] && c > 0) {
            flags[cpar[c]] = 0;
            atomicMax(&s_max, (int32_t)c);
        }
    __syncthreads();
    // labels n .. n + max cluster-row child that never appear as a parent
    for (int64_t c = t; c < C; c += blockDim.x)
        if (c > s_max) flags[c] = 0;
    __syncthreads();
    block_scan_excl(flags, C, &s_total);
    for (int64_t c = t; c < C; c += blockDim.x) {
        bool on = c <= s_max && (c + 1 < C ? flags[c + 1] - flags[c] : s_total - flags[c]) == 1;
        if (on) sel[flags[c]] = (int32_t)(n + c);
    }
    if (t == 0) *n_sel = s_max < 0 ? 0 : s_total;
}

// ---------------------------------------------------------------- labels
// Membership strength of a point that leaves at lambda lx a cluster whose
// largest point lambda is mx (cluster_trees.py:1011).
__device__ __forceinline__ float strength(float lx, float mx) {
    const double ml = (double)mx;
    if (ml == 0.0 || !isfinite(lx)) return 1.0f;
    const double lv = (double)lx < ml ? (double)lx : ml;
    return (float)(lv / ml);
}
__global__ void sel_flags_kernel(int64_t n_sel, int64_t n, int64_t C, const int32_t* __restrict__ sel,
                                 int8_t* __restrict__ is_sel, uint32_t* __restrict__ key,
                                 int32_t* __restrict__ val) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_sel) return;
    int32_t c = sel[i] - (int32_t)n;
    if (c >= 0 && c < C) is_sel[c] = 1;
    key[i] = (uint32_t)sel[i];
    val[i] = (int32_t)i;
}
__global__ void label_map_kernel(int64_t n_sel, int64_t n, int64_t C,
                                 const uint32_t* __restrict__ sorted_ids,
                                 int32_t* __restrict__ label_of, int32_t* __restrict__ by_label) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_sel) return;
    int32_t c = (int32_t)sorted_ids[j] - (int32_t)n;
    by_label[j] = c;
    if (c >= 0 && c < C) atomicMax(&label_of[c], (int32_t)j);  // last position wins
}
// Nearest selected cluster at or above every cluster (or the root), by pointer
// doubling, and the number of distinct selected clusters.  One block for up to
// kAncestorsBlock clusters: its log2(C) steps are a barrier each instead of a
// launch (all of the labels' work, by the block / by launches, us: 17,000
// clusters 246 / 240, 24,000 315 / 249, 1M 9,430 / 850).
constexpr int64_t kAncestorsBlock = 16384;
__global__ void __launch_bounds__(kEomThreads) ancestors_kernel(
    int64_t C, const int32_t* __restrict__ cpar, const int8_t* __restrict__ is_sel, int steps,
    int32_t* jmp, int32_t* sa, int32_t* jmp2, int32_t* sa2, int32_t* n_distinct) {
    int32_t mine = 0;
    for (int64_t c = threadIdx.x; c < C; c += blockDim.x) {
        jmp[c] = c == 0 ? 0 : (cpar[c] < 0 ? 0 : cpar[c]);
        sa[c] = (is_sel[c] || c == 0) ? (int32_t)c : -1;
        mine += is_sel[c] ? 1 : 0;
    }
    if (mine) atomicAdd(n_distinct, mine);
    __syncthreads();
    for (int r = 0; r < steps; ++r) {
        for (int64_t c = threadIdx.x; c < C; c += blockDim.x) {
            const int32_t a = jmp[c];
            jmp2[c] = jmp[a];
            sa2[c] = sa[c] != -1 ? sa[c] : sa[a];
        }
        __syncthreads();
        int32_t* t = jmp; jmp = jmp2; jmp2 = t;
        t = sa; sa = sa2; sa2 = t;
    }
}
// The same by launches over the whole GPU, where a block would read more
// clusters one after another than a launch costs.
__global__ void ancestors_init_kernel(int64_t C, const int32_t* __restrict__ cpar,
                                      const int8_t* __restrict__ is_sel, int32_t* __restrict__ jmp,
                                      int32_t* __restrict__ sa, int32_t* n_distinct) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = c < C && is_sel[c];
    if (c < C) {
        jmp[c] = c == 0 ? 0 : (cpar[c] < 0 ? 0 : cpar[c]);
        sa[c] = (on || c == 0) ? (int32_t)c : -1;
    }
    const unsigned b = __ballot_sync(kFull, on);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(n_distinct, __popc(b));
}
__global__ void ancestors_step_kernel(int64_t C, const int32_t* __restrict__ jmp,
                                      const int32_t* __restrict__ sa, int32_t* __restrict__ jmp2,
                                      int32_t* __restrict__ sa2) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int32_t a = jmp[c];
    jmp2[c] = jmp[a];
    sa2[c] = sa[c] != -1 ? sa[c] : sa[a];
}
// Label and membership strength of every point (probs_kernel's expression).
__global__ void point_labels_kernel(int64_t n, const int32_t* __restrict__ n_distinct, double eps,
                                    const int32_t* __restrict__ row_of_point,
                                    const int32_t* __restrict__ parent,
                                    const float* __restrict__ lam, const int32_t* __restrict__ sa,
                                    const int8_t* __restrict__ is_sel,
                                    const int32_t* __restrict__ label_of,
                                    const int32_t* __restrict__ by_label,
                                    const unsigned int* __restrict__ root_max,
                                    const unsigned int* __restrict__ death,
                                    int64_t* __restrict__ labels, float* __restrict__ probs,
                                    int* __restrict__ err) {
    int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n) return;
    int32_t r = row_of_point[x];
    int64_t lab = -1;
    float prob = 0.0f;
    if (r >= 0 && lam[r] != 0.0f) {
        int32_t a = sa[parent[r] - (int32_t)n];
        if (a != 0) {
            lab = label_of[a];
        } else if (*n_distinct == 1) {
            float lx = lam[r];
            bool take = eps > 0.0 ? ((double)lx >= 1.0 / eps) : (lx >= __uint_as_float(*root_max));
            if (take) {
                if (is_sel[0]) lab = label_of[0];
                else atomicOr(err, 1);
            }
        }
    }
    if (lab >= 0) prob = strength(lam[r], __uint_as_float(death[by_label[lab]]));
    labels[x] = lab;
    probs[x] = prob;
}
__global__ void probs_kernel(int64_t rows, int64_t n, const int32_t* __restrict__ child,
                             const float* __restrict__ lam, const int64_t* __restrict__ labels,
                             const int32_t* __restrict__ by_label,
                             const unsigned int* __restrict__ death, float* __restrict__ probs) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    int32_t x = child[r];
    if (x >= n) return;
    int64_t lab = labels[x];
    if (lab < 0) return;
    probs[x] = strength(lam[r], __uint_as_float(death[by_label[lab]]));
}
__global__ void fill_i64_kernel(int64_t* a, int64_t n, int64_t v) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = v;
}

#define LAUNCH(kernel, count, ...)                                          \
    do {                                                                    \
        if ((count) > 0) {                                                  \
            ::fhg::note_launch(); \
            kernel<<<grid_for((count), 256), 256, 0, s>>>(__VA_ARGS__);     \
            FHG_CUDA(cudaGetLastError());                                   \
        }                                                                   \
    } while (0)

// What the EOM selection needs beside LabelPre: rows grouped by parent and
// every cluster's score.
//
// The scores are one sequential float32 sum per cluster, so a large cluster's
// sum is a long chain of dependent additions on a single thread.  For many
// rows they are computed on a side stream while the stream lists the cluster
// rows and their parents; join() (also run by the destructor) orders the stream
// after them.  Every buffer the side stream touches belongs to the caller's
// Workspace, which outlives the join.
struct Prepared {
    int32_t *order = nullptr, *corder = nullptr, *ccnt = nullptr;
    uint32_t *key = nullptr, *cstart = nullptr;
    int64_t *start = nullptr, *end = nullptr;
    float *score = nullptr, *prod = nullptr;
    cudaStream_t main = nullptr, side = nullptr;
    cudaEvent_t done = nullptr;

    Prepared() = default;
    Prepared(const Prepared&) = delete;
    Prepared& operator=(const Prepared&) = delete;
    ~Prepared() { join(); }
    void join() {
        if (!side) return;
        cudaStreamWaitEvent(main, done, 0);
        cudaEventDestroy(done);
        cudaStreamDestroy(side);  // released once its work has completed
        side = nullptr;
        done = nullptr;
    }
};
// A stream and its events cost more than the sums of fewer rows.
constexpr int64_t kSideRows = 1 << 18;

// LabelPre of a tree; with P also what the EOM selection needs.
int prepare(Workspace& ws, const Condensed& ct, LabelPre* pre, Prepared* P) {
    cudaStream_t s = ws.stream();
    const int64_t C = ct.n_clusters, rows = ct.rows, n = ct.n;
    *pre = LabelPre();
    // all arrays that start as -1, then all that start as 0
    FHG_TRY(ws.alloc(&pre->row_of_point, (size_t)(n + 2 * C)));
    pre->row_of_cluster = pre->row_of_point + n;
    uint32_t* cstart = reinterpret_cast<uint32_t*>(pre->row_of_cluster + C);
    FHG_CUDA(cudaMemsetAsync(pre->row_of_point, 0xff, sizeof(int32_t) * (n + 2 * C), s));
    int64_t* zeroed;
    FHG_TRY(ws.alloc(&zeroed, (size_t)(3 * C + 1)));
    FHG_CUDA(cudaMemsetAsync(zeroed, 0, sizeof(int64_t) * (3 * C + 1), s));
    pre->death = reinterpret_cast<unsigned int*>(zeroed + 2 * C);
    int32_t* ccnt = reinterpret_cast<int32_t*>(pre->death + C);
    pre->root_max = reinterpret_cast<unsigned int*>(zeroed + 3 * C);
    FHG_TRY(ws.alloc(&pre->cpar, (size_t)C));
    FHG_TRY(ws.alloc(&pre->nsize, (size_t)C));
    FHG_TRY(ws.alloc(&pre->in_tree, (size_t)C));
    if (P) {
        P->start = zeroed;
        P->end = zeroed + C;
        P->ccnt = ccnt;
        P->cstart = cstart;
        FHG_TRY(ws.alloc(&P->key, (size_t)rows));
        FHG_TRY(ws.alloc(&P->order, (size_t)rows));
        FHG_TRY(ws.alloc(&P->prod, (size_t)rows));
        FHG_TRY(ws.alloc(&P->corder, (size_t)rows));
        FHG_TRY(ws.alloc(&P->score, (size_t)C));
    }
    ::fhg::note_launch();
    row_facts_kernel<<<grid_for(rows, kFactsThreads * kFactsRows), kFactsThreads, 0, s>>>(
        rows, n, ct.parent, ct.child, ct.lambda, ct.csize, pre->row_of_point, pre->row_of_cluster,
        pre->root_max, pre->death, P ? P->key : (uint32_t*)nullptr,
        P ? P->order : (int32_t*)nullptr);
    FHG_CUDA(cudaGetLastError());
    if (P) {
        FHG_TRY(radix_sort_u32(ws, P->key, P->order, rows, 0, bits_for(C)));
        LAUNCH(products_kernel, rows, rows, P->key, P->order, ct.lambda, ct.csize, P->prod,
               P->start, P->end);
        cudaStream_t ss = s;  // (the stream itself if no other can be made)
        cudaEvent_t fork = nullptr;
        if (rows < kSideRows) {
            P->side = nullptr;
        } else if (cudaStreamCreateWithFlags(&P->side, cudaStreamNonBlocking) == cudaSuccess) {
            if (cudaEventCreateWithFlags(&fork, cudaEventDisableTiming) == cudaSuccess &&
                cudaEventCreateWithFlags(&P->done, cudaEventDisableTiming) == cudaSuccess &&
                cudaEventRecord(fork, s) == cudaSuccess &&
                cudaStreamWaitEvent(P->side, fork, 0) == cudaSuccess) {
                ss = P->side;
                P->main = s;
            } else {
                if (P->done) cudaEventDestroy(P->done);
                P->done = nullptr;
                cudaStreamDestroy(P->side);
                P->side = nullptr;
            }
            if (fork) cudaEventDestroy(fork);
        } else {
            P->side = nullptr;
            cudaGetLastError();
        }
        if (C > 0) {
            if (rows >= kBigRows) {
                ::fhg::note_launch();
                score_big_kernel<<<(unsigned)(C < 1024 ? C : 1024), kScoreThreads, 0, ss>>>(
                    C, P->start, P->end, P->prod, pre->row_of_cluster, ct.lambda, ct.csize,
                    P->score);
                FHG_CUDA(cudaGetLastError());
            }
            ::fhg::note_launch();
            const bool many = C > kScoreWarps;
            (many ? score_many_kernel : score_kernel)<<<grid_for(C, many ? 256 : 8), 256, 0, ss>>>(
                C, P->start, P->end, P->prod, pre->row_of_cluster, ct.lambda, ct.csize, P->score);
            FHG_CUDA(cudaGetLastError());
        }
        if (P->side) FHG_CUDA(cudaEventRecord(P->done, P->side));
        FHG_TRY(compact(ws, ClusterRows{P->key, P->order, ct.csize, P->corder, P->cstart, P->ccnt},
                        rows, nullptr));
    }
    LAUNCH(cluster_info_kernel, C, C, n, pre->row_of_cluster, ct.parent, ct.csize, pre->cpar,
           pre->nsize, pre->in_tree);
    pre->ready = true;
    return FHG_OK;
}

}  // namespace

namespace {
__global__ void narrow_rows_kernel(int64_t rows, const int64_t* __restrict__ p,
                                   const int64_t* __restrict__ c, int32_t* __restrict__ op,
                                   int32_t* __restrict__ oc, unsigned long long* __restrict__ mx) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    op[r] = (int32_t)p[r];
    oc[r] = (int32_t)c[r];
    // labels fit 32 bits: combine the warp first, then one atomic per warp
    const unsigned act = __activemask();
    const unsigned m = __reduce_max_sync(act, (unsigned)max(p[r], c[r]));
    if ((int)(threadIdx.x & 31) == __ffs(act) - 1) atomicMax(mx, (unsigned long long)m);
}
}  // namespace

int condensed_from_arrays(Workspace& ws, const int64_t* parent, const int64_t* child,
                          const float* lambda, const float* csize, int64_t rows, Condensed* out) {
    cudaStream_t s = ws.stream();
    *out = Condensed();
    out->rows = rows;
    if (rows <= 0) return FHG_OK;
    unsigned long long* mx;
    FHG_TRY(ws.alloc(&out->parent, (size_t)rows));
    FHG_TRY(ws.alloc(&out->child, (size_t)rows));
    FHG_TRY(ws.alloc(&mx, 1));
    FHG_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned long long), s));
    LAUNCH(narrow_rows_kernel, rows, rows, parent, child, out->parent, out->child, mx);
    int64_t root = 0;
    unsigned long long hmx = 0;
    FHG_CUDA(cudaMemcpyAsync(&root, parent, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaMemcpyAsync(&hmx, mx, sizeof(hmx), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    out->n = root;
    out->n_clusters = (int64_t)hmx - root + 1;
    out->lambda = const_cast<float*>(lambda);
    out->csize = const_cast<float*>(csize);
    return FHG_OK;
}

int select_eom(Workspace& ws, const Condensed& ct, double max_cs, bool allow_single, int32_t* sel,
               int64_t* n_sel, LabelPre* pre) {
    cudaStream_t s = ws.stream();
    *n_sel = 0;
    if (ct.rows == 0) return FHG_OK;
    Stage stage(s, "select");
    LabelPre own;
    if (!pre) pre = &own;
    Prepared P;
    FHG_TRY(prepare(ws, ct, pre, &P));
    P.join();
    const int64_t C = ct.n_clusters;
    int32_t *depth, *depth2, *jmp, *jmp2, *dcount, *byd, *flags;
    double* ret;
    int8_t *chose, *blocked;
    int64_t* nsel_dev;
    FHG_TRY(ws.alloc(&depth, (size_t)C));
    FHG_TRY(ws.alloc(&depth2, (size_t)C));
    FHG_TRY(ws.alloc(&flags, (size_t)C));
    FHG_TRY(ws.alloc(&jmp, (size_t)C));
    FHG_TRY(ws.alloc(&jmp2, (size_t)C));
    FHG_TRY(ws.alloc(&dcount, (size_t)C + 2));
    FHG_TRY(ws.alloc(&byd, (size_t)C));
    FHG_TRY(ws.alloc(&ret, (size_t)C));
    FHG_TRY(ws.alloc(&chose, (size_t)C));
    FHG_TRY(ws.alloc(&blocked, (size_t)C));
    FHG_TRY(ws.alloc(&nsel_dev, 1));
    const bool here = C <= kEomShared;
    const size_t smem = here ? kEomBytes * (size_t)C + 16 : 0;
    FHG_CUDA(cudaFuncSetAttribute(eom_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kEomBytes * kEomShared + 16)));
    ::fhg::note_launch();
    (here ? eom_kernel<true> : eom_kernel<false>)<<<1, kEomThreads, smem, s>>>(
        C, pre->cpar, pre->nsize, pre->in_tree, P.score, P.cstart, P.ccnt, P.corder, ct.child,
        ct.n, max_cs, allow_single ? 1 : 0, depth, depth2, jmp, jmp2, dcount, byd, ret, chose,
        blocked, flags, sel, nsel_dev);
    FHG_CUDA(cudaGetLastError());
    FHG_CUDA(cudaMemcpyAsync(n_sel, nsel_dev, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    return FHG_OK;
}

int select_leaf(Workspace& ws, const Condensed& ct, int32_t* sel, int64_t* n_sel,
                LabelPre* pre) {
    cudaStream_t s = ws.stream();
    *n_sel = 0;
    if (ct.rows == 0) return FHG_OK;
    LabelPre own;
    if (!pre) pre = &own;
    FHG_TRY(prepare(ws, ct, pre, nullptr));
    int32_t* flags;
    int64_t* nsel_dev;
    FHG_TRY(ws.alloc(&flags, (size_t)ct.n_clusters));
    FHG_TRY(ws.alloc(&nsel_dev, 1));
    ::fhg::note_launch();
    leaf_kernel<<<1, kEomThreads, 0, s>>>(ct.n_clusters, ct.n, pre->cpar, pre->in_tree, flags, sel,
                                          nsel_dev);
    FHG_CUDA(cudaGetLastError());
    FHG_CUDA(cudaMemcpyAsync(n_sel, nsel_dev, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    return FHG_OK;
}

int label_points(Workspace& ws, const Condensed& ct, const int32_t* sel, int64_t n_sel,
                 double eps, int64_t* labels, float* probs, const LabelPre* pre_in) {
    cudaStream_t s = ws.stream();
    const int64_t n = ct.n, rows = ct.rows, C = ct.n_clusters;
    Stage stage(s, "labels");
    if (rows == 0 || n_sel == 0) {
        FHG_CUDA(cudaMemsetAsync(probs, 0, sizeof(float) * n, s));
        LAUNCH(fill_i64_kernel, n, labels, n, (int64_t)-1);
        return FHG_OK;
    }
    LabelPre own;
    const LabelPre* pre = pre_in;
    if (!pre || !pre->ready) {
        FHG_TRY(prepare(ws, ct, &own, nullptr));
        pre = &own;
    }
    int8_t* is_sel;
    int32_t *label_of, *by_label, *jmp, *sa, *jmp2, *sa2;
    uint32_t* key;
    int32_t* val;
    int* err;
    // [error flag, distinct selected clusters, is_sel], zeroed together
    FHG_TRY(ws.alloc(&err, (size_t)(2 + (C + 3) / 4)));
    int32_t* n_distinct = err + 1;
    is_sel = reinterpret_cast<int8_t*>(err + 2);
    FHG_TRY(ws.alloc(&label_of, (size_t)C));
    FHG_TRY(ws.alloc(&by_label, (size_t)n_sel));
    FHG_TRY(ws.alloc(&jmp, (size_t)C));
    FHG_TRY(ws.alloc(&sa, (size_t)C));
    FHG_TRY(ws.alloc(&jmp2, (size_t)C));
    FHG_TRY(ws.alloc(&sa2, (size_t)C));
    FHG_TRY(ws.alloc(&key, (size_t)n_sel));
    FHG_TRY(ws.alloc(&val, (size_t)n_sel));
    FHG_CUDA(cudaMemsetAsync(err, 0, 2 * sizeof(int) + C, s));
    FHG_CUDA(cudaMemsetAsync(label_of, 0xff, sizeof(int32_t) * C, s));
    LAUNCH(sel_flags_kernel, n_sel, n_sel, n, C, sel, is_sel, key, val);
    FHG_TRY(radix_sort_u32(ws, key, val, n_sel, 0, 32));
    LAUNCH(label_map_kernel, n_sel, n_sel, n, C, key, label_of, by_label);
    const int steps = bits_for(C) + 1;
    if (C <= kAncestorsBlock) {
        ::fhg::note_launch();
        ancestors_kernel<<<1, kEomThreads, 0, s>>>(C, pre->cpar, is_sel, steps, jmp, sa, jmp2, sa2,
                                                   n_distinct);
        FHG_CUDA(cudaGetLastError());
        if (steps & 1) std::swap(sa, sa2);
    } else {
        LAUNCH(ancestors_init_kernel, C, C, pre->cpar, is_sel, jmp, sa, n_distinct);
        for (int r = 0; r < steps; ++r) {
            LAUNCH(ancestors_step_kernel, C, C, jmp, sa, jmp2, sa2);
            std::swap(jmp, jmp2);
            std::swap(sa, sa2);
        }
    }
    LAUNCH(point_labels_kernel, n, n, n_distinct, eps, pre->row_of_point, ct.parent, ct.lambda,
           sa, is_sel, label_of, by_label, pre->root_max, pre->death, labels,
           probs, err);
    int h_err = 0;
    FHG_CUDA(cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    if (h_err) {
        set_error("a point resolved to the root cluster, which is not selected (the reference "
                  "raises KeyError here)");
        return FHG_ERR_INVALID;
    }
    return FHG_OK;
}

int membership_strengths(Workspace& ws, const Condensed& ct, const int32_t* sel, int64_t n_sel,
                         const int64_t* labels, float* probs) {
    cudaStream_t s = ws.stream();
    const int64_t n = ct.n, rows = ct.rows, C = ct.n_clusters;
    FHG_CUDA(cudaMemsetAsync(probs, 0, sizeof(float) * n, s));
    if (rows == 0 || n_sel == 0) return FHG_OK;
    int8_t* is_sel;
    int32_t *label_of, *by_label, *val;
    uint32_t* key;
    FHG_TRY(ws.alloc(&is_sel, (size_t)C));
    FHG_TRY(ws.alloc(&label_of, (size_t)C));
    FHG_TRY(ws.alloc(&by_label, (size_t)n_sel));
    FHG_TRY(ws.alloc(&key, (size_t)n_sel));
    FHG_TRY(ws.alloc(&val, (size_t)n_sel));
    LabelPre pre;
    FHG_TRY(prepare(ws, ct, &pre, nullptr));
    FHG_CUDA(cudaMemsetAsync(is_sel, 0, C, s));
    FHG_CUDA(cudaMemsetAsync(label_of, 0xff, sizeof(int32_t) * C, s));
    LAUNCH(sel_flags_kernel, n_sel, n_sel, n, C, sel, is_sel, key, val);
    FHG_TRY(radix_sort_u32(ws, key, val, n_sel, 0, 32));
    LAUNCH(label_map_kernel, n_sel, n_sel, n, C, key, label_of, by_label);
    LAUNCH(probs_kernel, rows, rows, n, ct.child, ct.lambda, labels, by_label, pre.death, probs);
    return FHG_OK;
}

}  // namespace fhg
