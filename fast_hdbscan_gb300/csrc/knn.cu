// Exact k-nearest-neighbour search (core distances), warp-cooperative.
//
// One warp owns one bucket of 32 index-consecutive query points (lane =
// query).  It first scans its own bucket -- which contains the queries
// themselves -- to get a tight k-th distance, then walks up the bucket tree to
// the root: at every ancestor it searches the sibling subtree depth-first
// (shared-memory stack; a node is entered when ANY lane's lower bound is
// within that lane's current k-th distance).  At a
// leaf the warp loads the bucket's points (one coalesced load per lane) and
// every lane collects those within its k-th distance.  Each lane keeps its
// sorted top-K list (squared distance, caller index) in registers: exact
// distance ties are broken without a memory access, and the index positions
// of the result are looked up once at the end.
//
// Ordering: (squared distance, caller index), ascending -- the reference's
// parallel_tree_query order with equal distances ordered by index.
// Replaces numba_kdtree.py:680-792 (tree_query_recursion, simple_heap_push,
// deheap_sort, parallel_tree_query).
#include "index.cuh"

namespace fhg {
namespace {

// Warps of a block: their shared memory stays within the static 48 KB.
template <int SP>
__host__ __device__ constexpr int knn_warps() { return SP <= 8 ? 4 : 2; }
// Buckets needed by at most this many lanes are scanned query by query, each
// lane with its own candidate; otherwise candidate by candidate, each lane for
// its own query.  (Two, four or eight lanes to a query instead, with shared
// counters for the queues: 13.3 against 13.2 ms at 10M x 3-D, 11.7 against 9.3
// at 2M x 5-D.)
constexpr int kTransposeMax = 16;
// Resident blocks asked of the register allocator: small lists get 80 registers
// (100 above four dimensions), which keeps 24 (20) warps per SM, at the price of
// a few spilled words at K = 16 (12 stored and 15 loaded a thread in 3-D); larger
// lists take what they need.
template <int DIM, int K>
constexpr int knn_min_blocks() { return K > 16 || DIM > 8 ? 1 : DIM <= 4 ? 6 : 5; }
// Candidates at a lane's k-th distance that come after its k-th entry never join
// its list.  A few of them cost least where they are queued and merged like the
// others, but among many equal points a bucket holds nothing else.  Scans query
// by query drop them where a queue would overflow; the others drop each of them
// for lists of up to 24 (2 % of the kernel at 10M x 3-D; for 64 it would be 7).
// 300 points 1,000 times each, k = 6 / 16 / 24 / 40, ms: 0.71 / 1.16 / 1.87 / 5.6
// by insertion one by one, 2.2 / 3.5 / 3.9 / 8.9 queued and merged, 0.93 / 1.20 /
// 1.55 / 4.6 here.  (20,000 equal points, k = 6 / 31: 2.5 / 7.2, 23 / 52, 6.1 /
// 9.4: every bucket before the query's replaces its whole list.)
constexpr int kDropLateMax = 24;
// A lane's queue of candidates not yet in its list (see knn_kernel): the fill
// at which the warp empties its queues, and the row stride (odd, in 8-byte
// words: no bank conflicts across lanes).
constexpr int kQueueFull = 16, kQueue = kQueueFull + 8, kQueueStride = kQueue + 1;

__device__ __forceinline__ unsigned long long pack_entry(float d, int32_t o) {
    return ((unsigned long long)__float_as_uint(d) << 32) | (uint32_t)o;
}
__device__ __forceinline__ float entry_dist(unsigned long long e) {
    return __uint_as_float((uint32_t)(e >> 32));
}
__device__ __forceinline__ int32_t entry_orig(unsigned long long e) { return (int32_t)(uint32_t)e; }

__device__ __forceinline__ void compare_exchange(unsigned long long& a, unsigned long long& b) {
    const bool swap = a > b;
    const unsigned long long lo = swap ? b : a;
    b = swap ? a : b;
    a = lo;
}
// Ascending sort of 8 keys (Batcher's odd-even merge sort, 19 exchanges).
__device__ __forceinline__ void sort8(unsigned long long* v) {
#define FHG_CE(i, j) compare_exchange(v[i], v[j])
    FHG_CE(0, 1); FHG_CE(2, 3); FHG_CE(4, 5); FHG_CE(6, 7);
    FHG_CE(0, 2); FHG_CE(1, 3); FHG_CE(4, 6); FHG_CE(5, 7);
    FHG_CE(1, 2); FHG_CE(5, 6);
    FHG_CE(0, 4); FHG_CE(1, 5); FHG_CE(2, 6); FHG_CE(3, 7);
    FHG_CE(2, 4); FHG_CE(3, 5);
    FHG_CE(1, 2); FHG_CE(3, 4); FHG_CE(5, 6);
#undef FHG_CE
}
// Merges the ascending v[8] into the ascending key[K], keeping the K smallest
// in order; out = min(out, every key left out).
template <int K>
__device__ __forceinline__ void merge8(unsigned long long (&key)[K],
                                       const unsigned long long* v, unsigned long long& out) {
    constexpr bool kPow2 = (K & (K - 1)) == 0;
    constexpr int M = kPow2 ? K : 32;  // K = 24 merges as 32
    unsigned long long c[M];
#pragma unroll
    for (int j = 0; j < K; ++j) c[j] = key[j];
    if constexpr (kPow2) {
        // the K smallest of key ++ reverse(v, +inf...) form a bitonic run
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            unsigned long long x = v[j];
            compare_exchange(c[K - 1 - j], x);
            out = x < out ? x : out;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) c[M - 1 - j] = v[j];
    }
#pragma unroll
    for (int stride = M / 2; stride > 0; stride >>= 1) {
#pragma unroll
        for (int i = 0; i < M; ++i)
            if ((i & stride) == 0) compare_exchange(c[i], c[i + stride]);
    }
#pragma unroll
    for (int j = 0; j < K; ++j) key[j] = c[j];
    if constexpr (!kPow2) out = c[K] < out ? c[K] : out;
}

// What bounds this kernel is instruction issue and, next to it, the latency of a
// walk: 65 % of the issue slots are busy at 4M x 3-D, k = 16; stalls are fixed
// latencies first, then loads.  A bucket's candidates within a lane's k-th
// distance go into that lane's queue in shared memory; when some lane's queue
// fills up, every lane sorts its queue eight at a time and merges it into its
// sorted list, by networks that run the same instructions on all lanes.
// (Inserting each candidate as it came made the warp wait for its busiest lane in
// every bucket: about 150 insertions per warp at 1M x 3-D, k = 16, where a lane
// inserts 41; now about 20 merges.)  Until its queue is emptied a lane's k-th
// distance is out of date, i.e. larger: it queues some more candidates, and no
// result changes.  Measured (one GB300, lists inserted one by one -> this): 10M x
// 3-D, k = 16: 15.3 -> 12.6 ms; 2M x 5-D, k = 11: 10.4 -> 9.2; 60k x 13-D, k = 11:
// 2.3 -> 1.7.  (All nodes of a level at once against the bucket's box, as the
// Boruvka search does: 16.1 ms at 10M -- one outlying query makes its bucket walk
// everything.)
template <int DIM, int SP, int K>
__global__ void __launch_bounds__(knn_warps<SP>() * 32, knn_min_blocks<DIM, K>())
    knn_kernel(IndexView ix, int k, float* __restrict__ d_s, int32_t* __restrict__ i_s,
               float* __restrict__ d_o, int32_t* __restrict__ i_o, int8_t* __restrict__ tie_s,
               int io_stride, int io_skip, const float* __restrict__ cap2,
               const uint8_t* __restrict__ redo, uint8_t* __restrict__ fail,
               unsigned long long* fail_count, unsigned long long* scan_count, int split) {
    constexpr int kKnnWarps = knn_warps<SP>();
    constexpr bool kDropLate = K <= kDropLateMax;
    __shared__ float4 s_cand[kKnnWarps][32 * (SP / 4)];
    __shared__ float4 s_query[kKnnWarps][32 * (SP / 4)];
    __shared__ int32_t s_corig[kKnnWarps][32];
    __shared__ unsigned long long s_queue[kKnnWarps][32 * kQueueStride];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // `split` warps share a bucket's queries, 32 / split each (knn_split).
    const int64_t part = (int64_t)blockIdx.x * kKnnWarps + warp;
    const int64_t leaf = part / split;
    if (leaf >= ix.nleaves) return;
    const int64_t qi = leaf * kLeaf + lane;
    const bool own_part = lane * split / 32 == (int)(part % split);
    // redo (nullable): only these queries search (the fallback of a capped
    // pass); cap2 (nullable): every query's list starts full of sentinels at
    // its squared search radius, so only points within it are considered.
    const bool valid = own_part && qi < ix.n && (!redo || redo[qi]);
    if (!__any_sync(kFull, valid)) return;
    float q[DIM];
    {
        float t[SP];
        if (valid) load_pt<SP>(ix.pts, qi, t);
        else
#pragma unroll
            for (int j = 0; j < SP; ++j) t[j] = 0.0f;
#pragma unroll
        for (int j = 0; j < DIM; ++j) q[j] = t[j];
#pragma unroll
        for (int h = 0; h < SP / 4; ++h)
            s_query[warp][lane * (SP / 4) + h] =
                make_float4(t[4 * h], t[4 * h + 1], t[4 * h + 2], t[4 * h + 3]);
    }
    __syncwarp();
    // Each list entry is one 64-bit key: squared distance bits above the
    // caller index.  Non-negative floats order like their bit patterns, so
    // one unsigned compare orders entries by (distance, caller index).
    // Slots [0, K-k) hold a 0 sentinel so that the live list has length k;
    // empty live slots hold (+inf, INT32_MAX).
    unsigned long long key[K];
    const unsigned long long kEmptyKey =
        pack_entry(cap2 && valid ? cap2[qi] : INFINITY, INT32_MAX);
#pragma unroll
    for (int j = 0; j < K; ++j) key[j] = (j < K - k) ? 0ull : kEmptyKey;
    float4* cand = s_cand[warp];
    int32_t* corig = s_corig[warp];
    unsigned long long* queue = s_queue[warp];
    const int32_t* __restrict__ orig = ix.orig;

    // Least key of a point examined but left out of the list: its distance
    // equals the final k-th exactly when another point ties with the k-th.
    // (A capped list's sentinels follow every queued point: as this minimum
    // one stands for "no point".)
    unsigned long long rejected = ~0ull;
    int waiting = 0;  // entries in this lane's queue
    float thr = valid ? entry_dist(key[K - 1]) : -1.0f;  // (no distance is within -1)
    int scans = 0;  // buckets this warp scanned

    // The walk: the home bucket first (it holds the queries themselves and
    // gives a tight k-th distance), then up to the root, searching at each
    // ancestor the sibling subtree depth first, pruned by lower bounds.
    // Subtrees' boxes overlap, so no ancestor box bounds the search; but near
    // subtrees come first, and a far sibling whose box is out of every lane's
    // reach costs a single box test.  Inside a sibling subtree the child
    // nearer the home bucket in index order goes first: the left child of a
    // subtree to the right of the home path, the right child of one to its
    // left.  Both children are tested when their parent is expanded; only
    // needed ones are followed, the nearer at once, the farther by way of the
    // stack (lane j holds entry j: at most one entry per level) or, for a
    // bucket, of `later` with its bounds.
    //
    // Every bucket is scanned, and every queue emptied, at one place in the
    // code each: with the scan and the merges inlined where they are needed,
    // the kernel ran out of the instruction cache (3.1 of 10 stall cycles per
    // instruction at 2M x 3-D, k = 16).
    const int64_t first_leaf_node = ix.slots - 1;
    int64_t x = first_leaf_node + leaf;
    int32_t stack = 0, later = -1;
    int sp = 0;
    bool right_side = false;
    float later_lb = 0.0f;
    // Slots past the last bucket have boxes without points, whose bound, +inf, is
    // within reach of a list that is not full yet, or holds points at infinite
    // (overflowed) distances: only then are nodes looked at for it.  (2^20 + 1
    // points, whose last bucket holds one, scanned every empty slot: 131 ms.)
    bool unfilled = true;
    auto empty = [&](int32_t v) {
        float b[2 * SP];
        load_box<SP>(ix.box, v, b);
        return box_empty<SP>(b);
    };
    int64_t lf = leaf;  // the bucket to scan, -1 when the walk has ended
    bool need = valid;
    for (bool home = true;; home = false) {
        // ---- scan: the bucket's candidates within the k-th distance of each
        // lane that needs it join that lane's queue
        const int64_t base = lf * kLeaf;
        const int cnt = lf < 0 ? 0 : (int)(ix.n - base < kLeaf ? ix.n - base : kLeaf);
        unsigned todo = lf < 0 ? 0u : __ballot_sync(kFull, need);
        // (the home bucket fills every list: its lanes go through it together)
        const bool by_query = !home && __popc(todo) <= kTransposeMax;
        float own[SP];  // this lane's candidate (lane t holds candidate t)
        int32_t own_o = 0;
#pragma unroll
        for (int j = 0; j < SP; ++j) own[j] = INFINITY;  // (within no distance but +inf)
        if (lane < cnt) {
            load_pt<SP>(ix.pts, base + lane, own);
            own_o = __ldg(orig + base + lane);
        }
        if (lf >= 0) ++scans;
        if (!by_query) {
            __syncwarp();
#pragma unroll
            for (int h = 0; h < SP / 4; ++h)
                cand[lane * (SP / 4) + h] =
                    make_float4(own[4 * h], own[4 * h + 1], own[4 * h + 2], own[4 * h + 3]);
            corig[lane] = own_o;
            __syncwarp();
        }
        const unsigned every = cnt >= 32 ? kFull : (1u << cnt) - 1u;
        unsigned left = 0;    // by_query: candidates this lane's query had no room for,
        bool again = false;   // and whether these are looked at now
        int t0 = 0;
        // the queues are emptied at a fill of kQueueFull; after the home
        // bucket and at the end always
        const int full = home || lf < 0 ? 1 : kQueueFull;
        for (;;) {
            bool room = true;  // false: a queue must be emptied to go on
            if (by_query) {
                // Few lanes need the bucket: each lane takes its own candidate
                // and the warp visits only the needing queries.  What a query's
                // queue has no room for waits until all queues are emptied.
                unsigned more = 0;
                while (todo) {
                    const int i = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    float y[SP];
#pragma unroll
                    for (int h = 0; h < SP / 4; ++h) {
                        const float4 v = s_query[warp][i * (SP / 4) + h];
                        y[4 * h] = v.x; y[4 * h + 1] = v.y; y[4 * h + 2] = v.z; y[4 * h + 3] = v.w;
                    }
                    const float lim = __shfl_sync(kFull, thr, i);
                    const float dd = rdist_rn<DIM>(y, own);
                    unsigned in = __ballot_sync(kFull, dd <= lim);
                    if (!in) continue;
                    in &= again ? __shfl_sync(kFull, left, i) : every;
                    const int have = __shfl_sync(kFull, waiting, i);
                    int place = have + __popc(in & ((1u << lane) - 1u));
                    if (have + __popc(in) > kQueue) {
                        // Many at once, mostly at equal distances: at the k-th only
                        // candidates before the k-th entry join, and what then has
                        // no room waits.
                        const int32_t last = __shfl_sync(kFull, entry_orig(key[K - 1]), i);
                        const unsigned late = __ballot_sync(kFull, dd == lim && own_o > last) & in;
                        in &= ~late;
                        place = have + __popc(in & ((1u << lane) - 1u));
                        const unsigned fit = __ballot_sync(kFull, place < kQueue) & in;
                        if (lane == i) {
                            left = in & ~fit;
                            if (late) rejected = min(rejected, pack_entry(lim, 0));
                        }
                        if (in != fit) more |= 1u << i;
                        in = fit;
                    }
                    if ((in >> lane) & 1u)
                        queue[i * kQueueStride + place] = pack_entry(dd, own_o);
                    if (lane == i) waiting += __popc(in);
                }
                todo = more;
                again = true;
                room = more == 0;
            } else {
                // Every lane reads candidate t from shared memory.
                const float lim = need ? thr : -1.0f;
                for (; t0 < cnt; t0 += 8) {
                    room = !__any_sync(kFull, waiting >= kQueueFull);
                    if (!room) break;
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int t = t0 + u;
                        float c[SP];
#pragma unroll
                        for (int h = 0; h < SP / 4; ++h) {
                            const float4 v = cand[t * (SP / 4) + h];
                            c[4 * h] = v.x; c[4 * h + 1] = v.y;
                            c[4 * h + 2] = v.z; c[4 * h + 3] = v.w;
                        }
                        const float dd = rdist_rn<DIM>(q, c);
                        if (dd <= lim && t < cnt) {
                            const unsigned long long e = pack_entry(dd, corig[t]);
                            queue[lane * kQueueStride + waiting] = e;
                            if (!kDropLate || dd < lim ||
                                entry_orig(e) < entry_orig(key[K - 1]))
                                ++waiting;
                            else
                                rejected = min(rejected, e);
                        }
                    }
                }
            }
            // ---- queues into lists
            if (!room || __any_sync(kFull, waiting >= full)) {
                __syncwarp();
                // whole eights of the fullest queue; the rest waits, unless the
                // lists are wanted now or one query needs all its room
                const int keep = full == 1 || (by_query && !room) ? 0 : 7;
                for (int most = __reduce_max_sync(kFull, waiting); most > keep; most -= 8) {
                    unsigned long long v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        v[j] = j < waiting ? queue[lane * kQueueStride + waiting - 1 - j] : ~0ull;
                    waiting = max(waiting - 8, 0);
                    sort8(v);
                    merge8<K>(key, v, rejected);
                }
                if (valid) thr = entry_dist(key[K - 1]);
                unfilled = __any_sync(kFull, thr == INFINITY);
                __syncwarp();
            }
            if (room) break;
        }
        if (lf < 0) break;

        // ---- on to the next bucket some lane needs
        lf = -1;
        if (later >= 0) {
            need = later_lb <= thr;
            if (__any_sync(kFull, need)) lf = later;
            later = -1;
        }
        while (lf < 0) {
            int32_t node;
            if (sp == 0) {
                if (x == 0) break;
                node = (int32_t)((x & 1) ? x + 1 : x - 1);
                right_side = (x & 1) != 0;
                x = (x - 1) >> 1;
                float b[2 * SP];
                load_box<SP>(ix.box, node, b);
                need = box_lb_n<DIM, SP>(b, q) <= thr;
                if (!__any_sync(kFull, need) || (unfilled && empty(node))) continue;
                if (node >= first_leaf_node) {
                    lf = node - first_leaf_node;
                    break;
                }
            } else {
                node = __shfl_sync(kFull, stack, --sp);
            }
            // down to a bucket, or until no child is needed
            for (;;) {
                const int32_t l = 2 * node + 1, r = l + 1;
                const int32_t nearc = right_side ? l : r, farc = right_side ? r : l;
                float bn[2 * SP], bf[2 * SP];
                load_box<SP>(ix.box, nearc, bn);
                load_box<SP>(ix.box, farc, bf);
                const float lbn = box_lb_n<DIM, SP>(bn, q), lbf = box_lb_n<DIM, SP>(bf, q);
                bool an = __any_sync(kFull, lbn <= thr), af = __any_sync(kFull, lbf <= thr);
                if (unfilled) {
                    an = an && !empty(nearc);
                    af = af && !empty(farc);
                }
                if (!an && !af) break;
                if (l >= first_leaf_node) {
                    lf = (an ? nearc : farc) - first_leaf_node;
                    need = (an ? lbn : lbf) <= thr;
                    if (an && af) {
                        later = farc - (int32_t)first_leaf_node;
                        later_lb = lbf;
                    }
                    break;
                }
                if (an && af) {
                    if (lane == sp) stack = farc;
                    ++sp;
                }
                node = an ? nearc : farc;
            }
        }
    }
    if (scan_count && lane == 0) atomicAdd(scan_count, (unsigned long long)scans);
    if (!valid) return;
    // Certification: a capped list whose k-th slot still holds a sentinel had
    // fewer than k points within the radius -- its query is searched again
    // without a cap.  A full list is the exact answer: every point closer than
    // its k-th entry lies within the radius and was considered.
    if (cap2 && entry_orig(key[K - 1]) == INT32_MAX) {
        fail[qi] = 1;
        if (fail_count) atomicAdd(fail_count, 1ull);
        return;
    }
    const float rejmin =
        rejected == ~0ull || entry_orig(rejected) == INT32_MAX ? INFINITY : entry_dist(rejected);
    if (tie_s) tie_s[qi] = rejmin == entry_dist(key[K - 1]) ? 1 : 0;
    const int64_t o_row = orig[qi];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        if (j < K - k) continue;
        const int jj = j - (K - k);
        const float dj = entry_dist(key[j]);
        const int32_t oj = entry_orig(key[j]);
        const int32_t o = oj == INT32_MAX ? -1 : oj;  // k > n leaves slots empty
        if (d_s) {
            d_s[qi * k + jj] = dj;
            i_s[qi * k + jj] = o >= 0 ? __ldg(ix.rank + o) : -1;
        }
        if (d_o) d_o[o_row * k + jj] = dj;
        if (i_o && jj >= io_skip) i_o[o_row * io_stride + jj - io_skip] = o;
    }
}

// ------------------------------------------------------------ longer lists
// k > 64 (the list no longer fits in registers): a warp per query.  Candidates
// below a threshold are appended to an unordered buffer in shared memory; when
// it is full it is cut back to between k and k + kCutSlack of its smallest
// keys, which gives the next threshold; what is left at the end is sorted
// once.  The tree is read 32 nodes at a time, a lane each: first the group of
// up to 32 buckets around the query's own, nearest bucket first, then the
// sibling subtrees on the way up.  A bucket is scanned while its box bound is
// within the threshold's distance, which is never below the k-th distance: the
// list is the k smallest keys of all points and the tie flag has knn_kernel's
// meaning, so both kernels give the same outputs bit for bit.
//
// What bounds it is instruction issue (75 % of the slots before).  Sorting each
// bucket's candidates and merging them into a sorted list took most of it, one
// node at a time most of the rest.  300k x 3-D, k = 101: 4.06 -> 1.88 ms
// (room for 64 / 96 / 160 / 256 keys between cuts: 2.11 / 1.95 / 1.88 / 1.93).
constexpr int kCutSlack = 8;
// An expansion leaves at most 31 nodes besides the one that goes on, and a tree
// of 2^26 buckets has four expansions on a path.
constexpr int kLargeStack = 5 * 32;
constexpr int kLargeGrowth = 160;  // what a buffer takes between two cuts, at least
__host__ __device__ constexpr int large_pow2(int k) {
    int p = 64;
    while (p < k) p *= 2;
    return p;
}
__host__ __device__ constexpr int large_cap(int k) {
    const int a = ((k + kCutSlack + 31) & ~31) + kLargeGrowth, b = large_pow2(k);
    return a > b ? a : b;
}

// Cuts a buffer of cnt > keep distinct keys back to its smallest, between keep
// and keep + slack of them, and lowers `below` to a key that these are below
// and the others are not; out = min(out, distance of each key left out).  The
// key is found by bitwise descent from the highest bit in which the buffer's
// extremes differ: the keys are distinct, so the number below a key grows by one
// at a time and the descent meets one within the slack; five or six bits do with
// some of it.
__device__ __forceinline__ int large_cut(unsigned long long* buf, int cnt, int keep, int slack,
                                         int lane, unsigned long long& below, float& out) {
    __syncwarp();
    unsigned long long lo = ~0ull, hi = 0ull;
    for (int e = lane; e < cnt; e += 32) {
        const unsigned long long v = buf[e];
        lo = v < lo ? v : lo;
        hi = v > hi ? v : hi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(kFull, lo, o);
        const unsigned long long b = __shfl_xor_sync(kFull, hi, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    const int top = 63 - __clzll((long long)(lo ^ hi));
    unsigned long long res = top < 63 ? lo & ~((2ull << top) - 1ull) : 0ull;
    bool settled = false;
    for (int b = top; b >= 0 && !settled; --b) {
        const unsigned long long trial = res | (1ull << b);
        int c = 0;
        for (int e = lane; e < cnt; e += 32) c += buf[e] < trial ? 1 : 0;
        c = __reduce_add_sync(kFull, c);
        if (c <= keep + slack) res = trial;
        settled = c >= keep && c <= keep + slack;
    }
    int at = 0;
    const unsigned lt = (1u << lane) - 1u;
    for (int e0 = 0; e0 < cnt; e0 += 32) {
        const unsigned long long v = e0 + lane < cnt ? buf[e0 + lane] : ~0ull;
        const bool on = v < res;
        if (!on && e0 + lane < cnt) out = fminf(out, entry_dist(v));
        const unsigned m = __ballot_sync(kFull, on);
        if (on) buf[at + __popc(m & lt)] = v;
        at += __popc(m);
        __syncwarp();
    }
    below = res;
    return at;
}

// Ascending bitonic sort of buf[0, m), m a power of two >= 64, by one warp.
__device__ __forceinline__ void large_sort(unsigned long long* buf, int m, int lane) {
    for (int size = 2; size <= m; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncwarp();
            for (int p = lane; p < m / 2; p += 32) {
                const int i = 2 * p - (p & (stride - 1)), j = i + stride;
                const unsigned long long x = buf[i], y = buf[j];
                if ((x > y) == ((i & size) == 0)) {
                    buf[i] = y;
                    buf[j] = x;
                }
            }
        }
    __syncwarp();
}

template <int DIM, int SP>
__global__ void __launch_bounds__(128) knn_large_kernel(IndexView ix, int k, int cap,
                                                        float* __restrict__ d_s,
                                                        int32_t* __restrict__ i_s,
                                                        float* __restrict__ d_o,
                                                        int32_t* __restrict__ i_o,
                                                        int8_t* __restrict__ tie_s, int io_stride,
                                                        int io_skip,
                                                        unsigned long long* scan_count) {
    extern __shared__ unsigned long long s_lists[];  // [warps][cap]
    __shared__ int32_t s_stack[4][kLargeStack];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t qi = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (qi >= ix.n) return;
    unsigned long long* buf = s_lists + (size_t)warp * cap;
    int32_t* st = s_stack[warp];
    float q[DIM];
    {
        float t[SP];
        load_pt<SP>(ix.pts, qi, t);
#pragma unroll
        for (int j = 0; j < DIM; ++j) q[j] = t[j];
    }
    unsigned long long below = pack_entry(INFINITY, INT32_MAX);  // only keys below it are wanted
    float rejmin = INFINITY;  // least distance of an examined point left out
    int cnt = 0, scans = 0;
    auto bound = [&](int64_t node) {
        float b[2 * SP];
        load_box<SP>(ix.box, node, b);
        return box_lb_n<DIM, SP>(b, q);
    };
    auto scan_leaf = [&](int64_t lf) {
        ++scans;
        const int64_t base = lf * kLeaf;
        const bool here = base + lane < ix.n;
        unsigned long long key = ~0ull;
        float dd = INFINITY;
        if (here) {
            float c[SP];
            load_pt<SP>(ix.pts, base + lane, c);
            dd = rdist_rn<DIM>(q, c);
            key = pack_entry(dd, __ldg(ix.orig + base + lane));
        }
        unsigned m = __ballot_sync(kFull, here && key < below);
        if (cnt + __popc(m) > cap) {
            cnt = large_cut(buf, cnt, k, kCutSlack, lane, below, rejmin);
            m = __ballot_sync(kFull, here && key < below);
        }
        const bool keep = (m >> lane) & 1u;
        if (keep) buf[cnt + __popc(m & ((1u << lane) - 1u))] = key;
        else if (here) rejmin = fminf(rejmin, dd);
        cnt += __popc(m);
    };
    // The 2^levels buckets under a node, nearest first while one is in reach.
    auto scan_group = [&](int64_t first_leaf, int levels) {
        const int64_t lf = first_leaf + lane;
        float lb = lane < (1 << levels) && lf < ix.nleaves ? bound(ix.slots - 1 + lf) : NAN;
        for (;;) {
            const bool in = lb <= entry_dist(below);  // (never for NaN)
            // (bounds are not negative: their bits are in their order)
            const uint32_t least = __reduce_min_sync(kFull, in ? __float_as_uint(lb) : ~0u);
            if (least == ~0u) break;
            const int pick = __ffs(__ballot_sync(kFull, in && __float_as_uint(lb) == least)) - 1;
            scan_leaf(first_leaf + pick);
            if (lane == pick) lb = NAN;
        }
    };

    const int depth = 63 - __clzll((long long)ix.slots);  // levels under the root
    const int gl = min(depth, 5);
    const int64_t leaf = qi / kLeaf;
    scan_group(leaf >> gl << gl, gl);
    // node x at height h: its leaves are [(x + 1) 2^h - slots, ...)
    int64_t x = ((ix.slots + leaf) >> gl) - 1;
    for (int h = gl; x > 0; ++h, x = (x - 1) >> 1) {
        const bool right = (x & 1) != 0;  // the sibling lies to the right
        int sp = 0;
        int64_t node = right ? x + 1 : x - 1;
        int height = h;
        // the sibling itself, then what the stack holds
        if (!(bound(node) <= entry_dist(below))) continue;
        for (;;) {
            if (height <= 5) {
                scan_group(((node + 1) << height) - ix.slots, height);
            } else {
                const int e = min(height - 5, 5);
                const int64_t child = ((node + 1) << e) - 1 + lane;
                const bool in = lane < (1 << e) && bound(child) <= entry_dist(below);
                const unsigned m = __ballot_sync(kFull, in);
                // the ones on the query's side on top
                const unsigned after =
                    right ? (lane < 31 ? m >> (lane + 1) : 0u) : m & ((1u << lane) - 1u);
                if (in) st[sp + __popc(after)] = (int32_t)child;
                sp += __popc(m);
                __syncwarp();
            }
            bool found = false;
            while (sp > 0 && !found) {
                node = st[--sp];
                found = bound(node) <= entry_dist(below);
            }
            if (!found) break;
            height = depth - (63 - __clzll((long long)(node + 1)));
            __syncwarp();
        }
    }

    const int m = large_pow2(k);
    if (cnt > m) cnt = large_cut(buf, cnt, k, m - k, lane, below, rejmin);
    for (int j = cnt + lane; j < m; j += 32) buf[j] = pack_entry(INFINITY, INT32_MAX);
    large_sort(buf, m, lane);
    for (int j = k + lane; j < cnt; j += 32) rejmin = fminf(rejmin, entry_dist(buf[j]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rejmin = fminf(rejmin, __shfl_xor_sync(kFull, rejmin, o));
    if (scan_count && lane == 0) atomicAdd(scan_count, (unsigned long long)scans);
    if (tie_s && lane == 0) tie_s[qi] = rejmin == entry_dist(buf[k - 1]) ? 1 : 0;
    const int64_t o_row = ix.orig[qi];
    for (int j = lane; j < k; j += 32) {
        const unsigned long long e = buf[j];
        const float dj = entry_dist(e);
        const int32_t oj = entry_orig(e);
        const int32_t o = oj == INT32_MAX ? -1 : oj;  // k > n leaves slots empty
        if (d_s) {
            d_s[qi * k + j] = dj;
            i_s[qi * k + j] = o >= 0 ? __ldg(ix.rank + o) : -1;
        }
        if (d_o) d_o[o_row * k + j] = dj;
        if (i_o && j >= io_skip) i_o[o_row * io_stride + j - io_skip] = o;
    }
}

template <int DIM>
int launch_knn_large(const fhg_index& ix, int k, float* d_s, int32_t* i_s, float* d_o,
                     int32_t* i_o, int8_t* tie_s, int io_stride, int io_skip, const KnnCap& cap,
                     cudaStream_t s) {
    constexpr int SP = DIM <= 4 ? 4 : (DIM <= 8 ? 8 : DIM);
    if (cap.cap2 || cap.redo) {
        set_error("knn: a search radius takes k <= 64 (got %d)", k);
        return FHG_ERR_UNSUPPORTED;
    }
    if (ix.n <= 0) return FHG_OK;
    // four warps a block (an SM holds 32 blocks, 64 warps), or one where four
    // buffers would not fit in the 48 KB that a block has without asking
    const size_t list = sizeof(unsigned long long) * (size_t)large_cap(k);
    const int warps = 4 * list <= 40 * 1024 ? 4 : 1;
    Stage stage(s, "knn_kernel");
    ::fhg::note_launch();
    knn_large_kernel<DIM, SP><<<grid_for(ix.n, warps), warps * 32, warps * list, s>>>(
        view_of(ix), k, large_cap(k), d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip,
        cap.scan_count);
    FHG_CUDA(cudaGetLastError());
    return FHG_OK;
}

// Warps per bucket.  A walk is one long dependent chain, so with few buckets
// its latency is the kernel's time (3,000 points, k = 16: 94 warps, 150 us of
// which a few per cent issue): the queries of a bucket then go to several
// warps, whose other lanes still share the work on candidates, until the GPU
// has 20 warps per SM.  Measured (us at 1 / 4 / 8 / 16 warps per bucket): 94
// buckets, 3-D, k = 16: 154 / 90 / 73 / 72; 313, 2-D: 123 / 91 / 79 / 82; 625,
// 5-D: 370 / 297 / 269 / 297; 1,875, 3-D, k = 31: 512 / 591 / 708 / 1,028.
constexpr int64_t kKnnWarpsWanted = 20 * 152;
int knn_split(int64_t nleaves) {
    int split = 1;
    while (split < 32 && 2 * split * nleaves <= kKnnWarpsWanted) split *= 2;
    return split;
}

template <int DIM, int K>
int launch_knn(const fhg_index& ix, int k, float* d_s, int32_t* i_s, float* d_o, int32_t* i_o,
               int8_t* tie_s, int io_stride, int io_skip, const KnnCap& cap, cudaStream_t s) {
    // padded width; for d > 8 the kernels run over all SP = DIM padded
    // coordinates (the padding is zero and adds exact zeros to distances)
    constexpr int SP = DIM <= 4 ? 4 : (DIM <= 8 ? 8 : DIM);
    constexpr int kKnnWarps = knn_warps<SP>();
    const int split = knn_split(ix.nleaves);
    const unsigned g = grid_for(ix.nleaves * split, kKnnWarps);
    Stage stage(s, "knn_kernel");
    ::fhg::note_launch();
    knn_kernel<DIM, SP, K><<<g, kKnnWarps * 32, 0, s>>>(view_of(ix), k, d_s, i_s, d_o, i_o,
                                                         tie_s, io_stride, io_skip, cap.cap2,
                                                         cap.redo, cap.fail, cap.fail_count,
                                                         cap.scan_count, split);
    FHG_CUDA(cudaGetLastError());
    return FHG_OK;
}

template <int DIM>
int dispatch_k(const fhg_index& ix, int k, float* d_s, int32_t* i_s, float* d_o, int32_t* i_o,
               int8_t* tie_s, int ios, int iok, const KnnCap& c, cudaStream_t s) {
    if (k <= 8) return launch_knn<DIM, 8>(ix, k, d_s, i_s, d_o, i_o, tie_s, ios, iok, c, s);
    if (k <= 16) return launch_knn<DIM, 16>(ix, k, d_s, i_s, d_o, i_o, tie_s, ios, iok, c, s);
    if (k <= 24) return launch_knn<DIM, 24>(ix, k, d_s, i_s, d_o, i_o, tie_s, ios, iok, c, s);
    if (k <= 32) return launch_knn<DIM, 32>(ix, k, d_s, i_s, d_o, i_o, tie_s, ios, iok, c, s);
    return launch_knn<DIM, 64>(ix, k, d_s, i_s, d_o, i_o, tie_s, ios, iok, c, s);
}

}  // namespace

int index_knn(const fhg_index& ix, int k, float* d_s, int32_t* i_s, float* d_o, int32_t* i_o,
              cudaStream_t s, int8_t* tie_s, int io_stride, int io_skip, const KnnCap& cap) {
    if (io_stride <= 0) io_stride = k;
    if (k < 1 || k > kKnnMaxK) {
        set_error("knn: k must be in [1, %d] (got %d)", kKnnMaxK, k);
        return k < 1 ? FHG_ERR_INVALID : FHG_ERR_UNSUPPORTED;
    }
    if ((d_s == nullptr) != (i_s == nullptr) || (d_o != nullptr && i_o == nullptr) ||
        (d_o != nullptr && (io_stride != k || io_skip != 0))) {
        set_error("knn: index-order outputs come in pairs; caller-order distances need ids");
        return FHG_ERR_INVALID;
    }
    Stage stage(s, "knn");
    if (k > 64) {  // the list no longer fits in registers
#define FHG_LARGE(D) launch_knn_large<D>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s)
        switch (ix.d) {
            case 1: return FHG_LARGE(1);
            case 2: return FHG_LARGE(2);
            case 3: return FHG_LARGE(3);
            case 4: return FHG_LARGE(4);
            case 5: return FHG_LARGE(5);
            case 6: return FHG_LARGE(6);
            case 7: return FHG_LARGE(7);
            case 8: return FHG_LARGE(8);
            default: return ix.d <= 16 ? FHG_LARGE(16) : FHG_LARGE(32);
        }
#undef FHG_LARGE
    }
    switch (ix.d) {
        case 1: return dispatch_k<1>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        case 2: return dispatch_k<2>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        case 3: return dispatch_k<3>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        case 4: return dispatch_k<4>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        case 5: return dispatch_k<5>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        case 6: return dispatch_k<6>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        case 7: return dispatch_k<7>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        case 8: return dispatch_k<8>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
        default:
            if (ix.d <= 16)
                return dispatch_k<16>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
            return dispatch_k<32>(ix, k, d_s, i_s, d_o, i_o, tie_s, io_stride, io_skip, cap, s);
    }
}

}  // namespace fhg
