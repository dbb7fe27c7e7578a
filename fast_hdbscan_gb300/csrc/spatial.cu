// Spatial index build: Hilbert keys -> radix sort -> median splits of chunks
// (low dimensions) -> bucketed points -> bottom-up bounding boxes.  Replaces
// the reference's single-threaded median-split KD-tree build
// (numba_kdtree.py:410-521); the tree here only serves as a pruning structure,
// so its shape does not affect results.
#include "index.cuh"
#include "primitives.cuh"

namespace fhg {
namespace {

constexpr int kBBThreads = 256;
constexpr int kBBBlocks = 304;  // partial bounding boxes: two blocks a SM
constexpr int kMaxDim = 32;  // bounding box layout: lo[0..32), hi[32..64)

// Per-block min/max of every dimension: partial[block][2][kMaxDim].  MAXD is
// 8 or kMaxDim; the loops are unrolled and predicated on d (no local memory).
template <int MAXD>
__global__ void bbox_partial_kernel(const float* __restrict__ X, int64_t n, int d,
                                    float* __restrict__ partial) {
    float lo[MAXD], hi[MAXD];
#pragma unroll
    for (int j = 0; j < MAXD; ++j) {
        lo[j] = INFINITY;
        hi[j] = -INFINITY;
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int j = 0; j < MAXD; ++j) {
            if (j < d) {
                float v = X[i * d + j];
                lo[j] = fminf(lo[j], v);
                hi[j] = fmaxf(hi[j], v);
            }
        }
    }
    __shared__ float s_lo[kBBThreads / 32][MAXD], s_hi[kBBThreads / 32][MAXD];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < MAXD; ++j) {
        float a = lo[j], b = hi[j];
        for (int o = 16; o; o >>= 1) {
            a = fminf(a, __shfl_xor_sync(kFull, a, o));
            b = fmaxf(b, __shfl_xor_sync(kFull, b, o));
        }
        if (lane == 0) {
            s_lo[w][j] = a;
            s_hi[w][j] = b;
        }
    }
    __syncthreads();
    if (threadIdx.x < MAXD) {
        float a = INFINITY, b = -INFINITY;
        for (int ww = 0; ww < kBBThreads / 32; ++ww) {
            a = fminf(a, s_lo[ww][threadIdx.x]);
            b = fmaxf(b, s_hi[ww][threadIdx.x]);
        }
        partial[blockIdx.x * 2 * kMaxDim + threadIdx.x] = a;
        partial[blockIdx.x * 2 * kMaxDim + kMaxDim + threadIdx.x] = b;
    }
}

// Hilbert key of at most 63 bits from a common-scale quantisation of all axes
// (bits per axis = min(63 / d, 31); at least one).  The quantised coordinates
// go through Skilling's axes-to-transpose map (J. Skilling, "Programming the
// Hilbert curve", 2004) and are then interleaved.
//
// Why Hilbert and not Morton: 32 consecutive points of a Morton order often
// straddle one of the curve's jumps, which leaves buckets with long boxes.  On
// 1M x 3-D points of widely varying density (k = 16) a warp's kNN walk scanned
// 44.5 buckets and tested 240 nodes in Morton order, 30.0 and 156 here; 500k x
// 5-D 209 -> 148 buckets, 60k x 24-D 218 -> 168.  D: the dimension (d <= 8),
// or kMaxDim with the loops predicated on d.
template <int D>
__global__ void hilbert_kernel(const float* __restrict__ X, int64_t n, int d,
                               const float* __restrict__ partial, int nb, int bits,
                               uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
    // the bounding box from the blocks' partial boxes
    __shared__ float s_lo[kMaxDim], s_hi[kMaxDim];
    if (threadIdx.x < 32) {
        for (int j = 0; j < d; ++j) {
            float a = INFINITY, b = -INFINITY;
            for (int t = threadIdx.x; t < nb; t += 32) {
                a = fminf(a, partial[t * 2 * kMaxDim + j]);
                b = fmaxf(b, partial[t * 2 * kMaxDim + kMaxDim + j]);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                a = fminf(a, __shfl_xor_sync(kFull, a, o));
                b = fmaxf(b, __shfl_xor_sync(kFull, b, o));
            }
            if (threadIdx.x == 0) {
                s_lo[j] = a;
                s_hi[j] = b;
            }
        }
    }
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    constexpr bool kExact = D <= 8;  // d == D
    float ext = 0.0f;
#pragma unroll
    for (int j = 0; j < D; ++j)
        if (kExact || j < d) ext = fmaxf(ext, s_hi[j] - s_lo[j]);
    const float qmax = (float)((1ull << bits) - 1ull);
    const uint32_t top = (uint32_t)((1ull << bits) - 1ull);
    const float scale = ext > 0.0f ? qmax / ext : 0.0f;
    uint32_t x[D];
#pragma unroll
    for (int j = 0; j < D; ++j) {
        x[j] = 0;
        if (kExact || j < d) {
            float t = (X[i * d + j] - s_lo[j]) * scale;
            t = fminf(fmaxf(t, 0.0f), qmax);
            x[j] = min((uint32_t)t, top);
        }
    }
    for (int b = bits - 1; b > 0; --b) {
        const uint32_t low = (1u << b) - 1u;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            if (kExact || j < d) {
                // bit b of axis j set: invert the low bits of axis 0; else
                // exchange the low bits of axes 0 and j
                const bool set = (x[j] >> b) & 1u;
                const uint32_t t = set ? 0u : (x[0] ^ x[j]) & low;
                x[0] ^= set ? low : t;
                x[j] ^= t;
            }
        }
    }
    uint32_t last = 0;
#pragma unroll
    for (int j = 1; j < D; ++j)
        if (kExact || j < d) x[j] ^= x[j - 1];
#pragma unroll
    for (int j = 0; j < D; ++j)
        if (kExact || j < d) last = x[j];
    uint32_t t = 0;
    for (int b = bits - 1; b > 0; --b)
        if ((last >> b) & 1u) t ^= (1u << b) - 1u;
    uint64_t key = 0;
    for (int b = bits - 1; b >= 0; --b) {
#pragma unroll
        for (int j = 0; j < D; ++j)
            if (kExact || j < d) key = (key << 1) | (((x[j] ^ t) >> b) & 1u);
    }
    keys[i] = key;
    vals[i] = (int32_t)i;
}

// Order-preserving map of float bits to uint32 and back.
__device__ __forceinline__ uint32_t ordered(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float unordered(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? u & 0x7fffffffu : ~u);
}

// One block per chunk of 2,048 (1,024 for d = 4, 5) consecutive positions of
// the curve order: with KD, the chunk is split further, then its points, ranks
// and boxes up to the chunk's root are written.
//
// The split: halves of 1,024, 512, ... 32 points along the axis of largest
// extent of each part, so that every node of the bucket tree below the chunk
// is an exact median split.  The median is found by bitwise descent on the
// ordered coordinate bits: a part of up to 128 points belongs to one warp
// (4 points a lane) and counts with ballots alone; larger parts add their
// warps' counts in shared memory, one barrier per bit, starting at the
// highest bit in which the part's extremes differ.  Points keep their order
// inside each half, and the points at the median fill the left half in that
// order: a fixed permutation of the input.
// Measured with the curve together (one GB300, Morton buckets -> this): 10M x
// 3-D, k = 16, kNN 22.2 -> 15.3 ms, Boruvka search 25.0 -> 15.2 ms, the build
// 2.1 -> 2.9 ms; 2M x 5-D, k = 11, 15.6 -> 10.4, 14.4 -> 9.8 and 0.7 -> 0.8.
// Walk cost (simulated, per warp, as above): 1M x 3-D 30.0 -> 24.1 buckets
// and 156 -> 128 node tests; 500k x 5-D 148 -> 129 buckets.  From 6
// dimensions on it gains nothing (13-D 159 -> 314 buckets, as the
// cuts along the few longest axes mix blobs and noise), so d <= kKdMaxDim.
// The chunk's coordinates stay in shared memory within the static 48 KB, which
// sets its size (500k x 5-D: 512, 1,024 and 2,048 points give 128.8, 128 and
// 128.8 buckets).
constexpr int kPer = 4;               // positions of a lane, 32 apart
constexpr int kWarpSpan = 32 * kPer;  // consecutive positions of a warp
constexpr int kKdMaxDim = 5;
__host__ __device__ constexpr int chunk_points(int d) { return d == 4 || d == 5 ? 1024 : 2048; }

template <int D>
__device__ __forceinline__ void kd_split(uint32_t (*sx)[chunk_points(D)], uint16_t* ia,
                                         uint16_t* ib, int cnt) {
    constexpr int kChunk = chunk_points(D), kChunkThreads = kChunk / kPer;
    constexpr int kParts = kChunk / (2 * kWarpSpan);  // most parts of several warps
    __shared__ uint32_t s_lo[kParts][D], s_hi[kParts][D];
    __shared__ int s_cnt[32][kParts];
    __shared__ int s_less[kChunkThreads / 32], s_eq[kChunkThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint16_t *cur = ia, *nxt = ib;
    for (int half = kChunk / 2; half >= kLeaf; half >>= 1) {
        const int seg = 2 * half;
        if (half >= cnt) continue;  // every part fits its left half
        const bool wide = seg > kWarpSpan;  // the part spans several warps
        if (wide) {
            const int nseg = kChunk / seg;
            if (tid < nseg * D) {
                s_lo[tid / D][tid % D] = 0xffffffffu;
                s_hi[tid / D][tid % D] = 0u;
            }
            for (int i = tid; i < 32 * nseg; i += kChunkThreads) s_cnt[i / nseg][i % nseg] = 0;
            __syncthreads();
        }
        // groups: the runs of this warp's 32-position rows that one part holds
        const int rows = wide ? kPer : seg / 32;
#pragma unroll
        for (int g = 0; g < kPer; ++g) {
            if (g * rows >= kPer) break;
            const int r0 = g * rows;
            const int start = ((w * kWarpSpan + r0 * 32) / seg) * seg;  // the part's first position
            const int have = min(cnt - start, seg);                    // its points
            uint32_t id[kPer], key[kPer];
            bool ok[kPer];
            uint32_t lo[D], hi[D];
#pragma unroll
            for (int j = 0; j < D; ++j) {
                lo[j] = 0xffffffffu;
                hi[j] = 0u;
            }
#pragma unroll
            for (int t = 0; t < kPer; ++t) {
                const int pos = w * kWarpSpan + (r0 + t) * 32 + lane;
                ok[t] = t < rows && pos < cnt;
                id[t] = ok[t] ? cur[pos] : 0u;
                if (ok[t]) {
#pragma unroll
                    for (int j = 0; j < D; ++j) {
                        const uint32_t v = sx[j][id[t]];
                        lo[j] = min(lo[j], v);
                        hi[j] = max(hi[j], v);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < D; ++j) {
                lo[j] = __reduce_min_sync(kFull, lo[j]);
                hi[j] = __reduce_max_sync(kFull, hi[j]);
            }
            const int sg = start / seg;
            if (wide) {
                if (lane == 0 && have > 0) {
#pragma unroll
                    for (int j = 0; j < D; ++j) {
                        atomicMin(&s_lo[sg][j], lo[j]);
                        atomicMax(&s_hi[sg][j], hi[j]);
                    }
                }
                __syncthreads();
#pragma unroll
                for (int j = 0; j < D; ++j) {
                    lo[j] = s_lo[sg][j];
                    hi[j] = s_hi[sg][j];
                }
            }
            int axis = 0;
            uint32_t alo = lo[0], ahi = hi[0];
            float ext = unordered(hi[0]) - unordered(lo[0]);
#pragma unroll
            for (int j = 1; j < D; ++j) {
                const float e = unordered(hi[j]) - unordered(lo[j]);
                if (e > ext) {
                    ext = e;
                    axis = j;
                    alo = lo[j];
                    ahi = hi[j];
                }
            }
#pragma unroll
            for (int t = 0; t < kPer; ++t) key[t] = ok[t] ? sx[axis][id[t]] : 0xffffffffu;
            // the value of rank `half` (1-based): its leading bits are the
            // extremes' common ones
            const bool split = have > half;
            uint32_t med = alo;
            if (split || wide) {
                const uint32_t diff = split ? alo ^ ahi : 0u;
                const int top = diff ? 31 - __clz(diff) : -1;
                if (top >= 0) med = alo & ~((2u << top) - 1u);
                if (!split || top < 0) med = alo;
                // wide parts of one level run the same number of steps
                for (int b = wide ? 31 : top; b >= 0; --b) {
                    if (wide && __syncthreads_and(b > top)) continue;
                    const uint32_t trial = med | (1u << b);
                    int c = 0;
#pragma unroll
                    for (int t = 0; t < kPer; ++t)
                        if (t < rows) c += __popc(__ballot_sync(kFull, ok[t] && key[t] < trial));
                    if (wide) {
                        if (lane == 0 && c) atomicAdd(&s_cnt[b][sg], c);
                        __syncthreads();
                        c = s_cnt[b][sg];
                    }
                    if (b <= top && c < half) med = trial;
                }
            }
            // places: everything below the median, then as many points at the
            // median as the left half still takes, in their order
            int less = 0, eq = 0;
            unsigned bl[kPer], be[kPer];
#pragma unroll
            for (int t = 0; t < kPer; ++t) {
                bl[t] = be[t] = 0u;
                if (t < rows) {
                    bl[t] = __ballot_sync(kFull, ok[t] && key[t] < med);
                    be[t] = __ballot_sync(kFull, ok[t] && key[t] == med);
                }
                less += __popc(bl[t]);
                eq += __popc(be[t]);
            }
            int less0 = 0, eq0 = 0, less_all = less;
            if (wide) {
                if (lane == 0) {
                    s_less[w] = less;
                    s_eq[w] = eq;
                }
                __syncthreads();
                less_all = 0;
                const int w0 = start / kWarpSpan, w1 = (start + seg) / kWarpSpan;
                for (int ww = w0; ww < w1; ++ww) {
                    const int a = s_less[ww], b = s_eq[ww];
                    if (ww < w) {
                        less0 += a;
                        eq0 += b;
                    }
                    less_all += a;
                }
            }
            const int need = half - less_all;
            const unsigned lt = (1u << lane) - 1u;
#pragma unroll
            for (int t = 0; t < kPer; ++t) {
                if (ok[t]) {
                    const int pos = w * kWarpSpan + (r0 + t) * 32 + lane;
                    const int lb = less0 + __popc(bl[t] & lt), eb = eq0 + __popc(be[t] & lt);
                    const int left_before = lb + min(eb, need);
                    const bool left = key[t] < med || (key[t] == med && eb < need);
                    const int dst = !split ? pos
                                    : left ? start + left_before
                                           : start + half + (pos - start - left_before);
                    nxt[dst] = (uint16_t)id[t];
                }
                less0 += __popc(bl[t]);
                eq0 += __popc(be[t]);
            }
        }
        __syncthreads();
        uint16_t* x = cur;
        cur = nxt;
        nxt = x;
    }
    if (cur != ia) {
        for (int i = tid; i < cnt; i += kChunkThreads) ia[i] = cur[i];
        __syncthreads();
    }
}

// Nodes of one kind from their children: (lo, hi) corners of 2 * P floats.
template <int P>
__device__ __forceinline__ void join_boxes(const float* l, const float* r, float* o) {
#pragma unroll
    for (int j = 0; j < P; ++j) {
        o[j] = fminf(l[j], r[j]);
        o[P + j] = fmaxf(l[P + j], r[P + j]);
    }
}

// iota: the caller's order is the curve order (one chunk with KD: no curve is
// needed).  Empty slots of the tree get empty boxes.
template <int D, int P, bool KD>
__global__ void __launch_bounds__(chunk_points(D) / kPer) chunk_kernel(
    const float* __restrict__ X, int64_t n, int d, int64_t slots, int iota,
    int32_t* __restrict__ orig, float* __restrict__ pts, int32_t* __restrict__ rank,
    float* __restrict__ box) {
    constexpr int kChunk = chunk_points(D), kChunkThreads = kChunk / kPer;
    constexpr int kChunkLeaves = kChunk / kLeaf;
    __shared__ uint32_t s_x[KD ? D : 1][KD ? kChunk : 1];
    __shared__ int32_t s_orig[kChunk];
    __shared__ uint16_t s_ia[KD ? kChunk : 1], s_ib[KD ? kChunk : 1];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int64_t base = (int64_t)blockIdx.x * kChunk;
    const int cnt = (int)max((int64_t)0, min(n - base, (int64_t)kChunk));
    for (int i = tid; i < cnt; i += kChunkThreads) {
        const int32_t o = iota ? (int32_t)(base + i) : orig[base + i];
        s_orig[i] = o;
        if constexpr (KD) {
#pragma unroll
            for (int j = 0; j < D; ++j) s_x[j][i] = ordered(X[(int64_t)o * D + j]);
            s_ia[i] = (uint16_t)i;
        }
    }
    __syncthreads();
    if constexpr (KD) kd_split<D>(s_x, s_ia, s_ib, cnt);
    // points and ranks, then one warp per bucket for its box
    const int leaves = (int)min(slots, (int64_t)kChunkLeaves);
    const int64_t first = slots - 1 + (int64_t)blockIdx.x * kChunkLeaves;
    for (int lf = w; lf < leaves; lf += kChunkThreads / 32) {
        const int i = lf * kLeaf + lane;
        const bool valid = i < cnt;
        float v[P];
#pragma unroll
        for (int j = 0; j < P; ++j) v[j] = 0.0f;
        if (valid) {
            const int src = KD ? s_ia[i] : i;
            const int32_t o = s_orig[src];
            if constexpr (KD) {
#pragma unroll
                for (int j = 0; j < D; ++j) v[j] = unordered(s_x[j][src]);
                orig[base + i] = o;
            } else {
#pragma unroll
                for (int j = 0; j < P; ++j)
                    if (j < d) v[j] = X[(int64_t)o * d + j];
            }
            float4* dst = reinterpret_cast<float4*>(pts) + (base + i) * (P / 4);
#pragma unroll
            for (int h = 0; h < P / 4; ++h)
                dst[h] = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
            rank[o] = (int32_t)(base + i);
        }
        const bool any = lf * kLeaf < cnt;
        float* out = box + (first + lf) * 2 * P;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            float a = valid ? v[j] : INFINITY, b = valid ? v[j] : -INFINITY;
            if (any) {
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    a = fminf(a, __shfl_xor_sync(kFull, a, o));
                    b = fmaxf(b, __shfl_xor_sync(kFull, b, o));
                }
            }
            if (lane == 0) {
                out[j] = a;
                out[P + j] = b;
            }
        }
    }
    // the levels above, up to the chunk's root
    int64_t level = slots - 1;  // first node of the level below
    for (int width = leaves / 2; width >= 1; width >>= 1) {
        __syncthreads();
        level = (level - 1) / 2;
        if (tid < width) {
            const int64_t node = level + (int64_t)blockIdx.x * width + tid;
            join_boxes<P>(box + (2 * node + 1) * 2 * P, box + (2 * node + 2) * 2 * P,
                          box + node * 2 * P);
        }
    }
}

// The levels above the chunks' roots: each block joins kTop consecutive nodes
// of the level of `width` nodes up to their common root (one block when width
// <= kTop), so a tree of up to 2^22 buckets takes two launches.
constexpr int kTop = 512;
template <int P>
__global__ void __launch_bounds__(kTop / 2) top_box_kernel(float* __restrict__ box, int64_t width) {
    const int span = (int)min(width, (int64_t)kTop);
    int64_t level = width - 1;
    for (int wd = span / 2; wd >= 1; wd >>= 1) {
        level = (level - 1) / 2;
        if (threadIdx.x < wd) {
            const int64_t node = level + (int64_t)blockIdx.x * wd + threadIdx.x;
            join_boxes<P>(box + (2 * node + 1) * 2 * P, box + (2 * node + 2) * 2 * P,
                          box + node * 2 * P);
        }
        __syncthreads();
    }
}

template <int D, int P, bool KD>
int fill_tree(fhg_index* ix, const float* X, bool iota, cudaStream_t s) {
    constexpr int leaves = chunk_points(D) / kLeaf;
    const int64_t chunks = (ix->slots + leaves - 1) / leaves;
    ::fhg::note_launch();
    chunk_kernel<D, P, KD><<<(unsigned)chunks, chunk_points(D) / kPer, 0, s>>>(
        X, ix->n, ix->d, ix->slots, iota ? 1 : 0, ix->orig, ix->pts, ix->rank, ix->box);
    FHG_CUDA(cudaGetLastError());
    for (int64_t width = chunks; width > 1;) {
        const int64_t blocks = (width + kTop - 1) / kTop;
        ::fhg::note_launch();
        top_box_kernel<P><<<(unsigned)blocks, kTop / 2, 0, s>>>(ix->box, width);
        FHG_CUDA(cudaGetLastError());
        width = blocks;
    }
    return FHG_OK;
}

// Points, ranks and boxes from the curve order in ix->orig.
int fill_tree(fhg_index* ix, const float* X, bool iota, cudaStream_t s) {
    switch (ix->d) {
        case 1: return fill_tree<1, 4, true>(ix, X, iota, s);
        case 2: return fill_tree<2, 4, true>(ix, X, iota, s);
        case 3: return fill_tree<3, 4, true>(ix, X, iota, s);
        case 4: return fill_tree<4, 4, true>(ix, X, iota, s);
        case 5: return fill_tree<5, 8, true>(ix, X, iota, s);
        default: break;
    }
    if (ix->d <= 8) return fill_tree<8, 8, false>(ix, X, iota, s);
    if (ix->d <= 16) return fill_tree<16, 16, false>(ix, X, iota, s);
    return fill_tree<32, 32, false>(ix, X, iota, s);
}

// One allocation holds the four arrays.
int index_alloc(fhg_index* ix, cudaStream_t s) {
    cudaMemPool_t pool;
    FHG_TRY(device_pool(&pool));
    auto room = [](int64_t bytes) { return (size_t)((bytes + 16 + 255) / 256 * 256); };
    const size_t pts = room((int64_t)sizeof(float) * ix->n * ix->pad);
    const size_t ids = room((int64_t)sizeof(int32_t) * ix->n);
    const size_t box = room((int64_t)sizeof(float) * ix->nnodes * 2 * ix->pad);
    char* base = nullptr;
    FHG_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&base), pts + 2 * ids + box, pool, s));
    ix->base = base;
    ix->pts = reinterpret_cast<float*>(base);
    ix->orig = reinterpret_cast<int32_t*>(base + pts);
    ix->rank = reinterpret_cast<int32_t*>(base + pts + ids);
    ix->box = reinterpret_cast<float*>(base + pts + 2 * ids);
    return FHG_OK;
}

// ix->orig = the points in Hilbert order.
int curve_order(fhg_index* ix, const float* X, cudaStream_t s) {
    const int64_t n = ix->n;
    const int d = ix->d;
    Workspace ws(s);
    float* partial;
    uint64_t* keys;
    const int nb = (int)std::min<int64_t>(kBBBlocks, (n + kBBThreads - 1) / kBBThreads);
    FHG_TRY(ws.alloc(&partial, (size_t)nb * 2 * kMaxDim));
    FHG_TRY(ws.alloc(&keys, (size_t)n));
    ::fhg::note_launch();
    if (d <= 8) bbox_partial_kernel<8><<<nb, kBBThreads, 0, s>>>(X, n, d, partial);
    else bbox_partial_kernel<kMaxDim><<<nb, kBBThreads, 0, s>>>(X, n, d, partial);
    FHG_CUDA(cudaGetLastError());
    const int bits = std::max(1, std::min(63 / d, 31));
    const unsigned g = grid_for(n, 256);
    ::fhg::note_launch();
#define FHG_HILBERT(D) hilbert_kernel<D><<<g, 256, 0, s>>>(X, n, d, partial, nb, bits, keys, ix->orig)
    switch (d) {
        case 1: FHG_HILBERT(1); break;
        case 2: FHG_HILBERT(2); break;
        case 3: FHG_HILBERT(3); break;
        case 4: FHG_HILBERT(4); break;
        case 5: FHG_HILBERT(5); break;
        case 6: FHG_HILBERT(6); break;
        case 7: FHG_HILBERT(7); break;
        case 8: FHG_HILBERT(8); break;
        default: FHG_HILBERT(kMaxDim); break;
    }
#undef FHG_HILBERT
    FHG_CUDA(cudaGetLastError());
    return radix_sort_u64(ws, keys, ix->orig, n, 0, bits * d);
}

}  // namespace

int index_free(fhg_index* ix, cudaStream_t s) {
    if (!ix) return FHG_OK;
    if (ix->base) cudaFreeAsync(ix->base, s);
    delete ix;
    return FHG_OK;
}

int index_build(const float* X, int64_t n, int32_t d, cudaStream_t s, fhg_index** out) {
    *out = nullptr;
    if (n < 1 || d < 1 || d > kMaxDim) {
        set_error("index_build: need n >= 1 and 1 <= d <= 32 (got n=%lld, d=%d)", (long long)n, d);
        return FHG_ERR_INVALID;
    }
    if (n >= ((int64_t)1 << 31) - 64) {
        set_error("index_build: n must be below 2^31");
        return FHG_ERR_INVALID;
    }
    Stage stage(s, "index_build");
    fhg_index* ix = new fhg_index();
    ix->n = n;
    ix->d = d;
    ix->pad = d <= 4 ? 4 : (d <= 8 ? 8 : (d <= 16 ? 16 : 32));
    ix->nleaves = (n + kLeaf - 1) / kLeaf;
    ix->slots = 1;
    while (ix->slots < ix->nleaves) ix->slots *= 2;
    ix->nnodes = 2 * ix->slots - 1;
    int rc = index_alloc(ix, s);
    if (rc != FHG_OK) {
        index_free(ix, s);
        return rc;
    }
    // one chunk that is split as a whole needs no curve order
    const bool iota = d <= kKdMaxDim && n <= chunk_points(d);
    if (!iota) rc = curve_order(ix, X, s);
    if (rc == FHG_OK) rc = fill_tree(ix, X, iota, s);
    if (rc != FHG_OK) {
        index_free(ix, s);
        return rc;
    }
    *out = ix;
    return FHG_OK;
}

}  // namespace fhg
