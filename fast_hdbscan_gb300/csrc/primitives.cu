// Exclusive scan and LSD radix sort (8-bit digits, stable) for sm_103a.
//
// Radix sort: one kernel counts every digit of every key, then one kernel per
// digit ranks, places and writes its tiles.  A tile learns how many items of
// each digit lie in the tiles before it from the words those tiles publish
// (decoupled look-back, D. Merrill and M. Garland, "Single-pass Parallel Prefix
// Scan with Decoupled Look-back", 2016: their own count first, then the count up
// to and including them).  Tiles are numbered as blocks start, so every tile before
// a running one has started; a wait that still goes on too long ends with the
// block counting the keys of the tiles before it itself.
//
// Scan: the sums of tiles, then every block adds up the sums before its tile.
#include <algorithm>
#include <type_traits>

#include "primitives.cuh"

namespace fhg {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanIPT = 4;
constexpr int kScanTile = kScanThreads * kScanIPT;

template <class T>
__device__ T block_exclusive_scan(T v, T* total) {
    __shared__ T warp_sums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        T w = lane < nw ? warp_sums[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(kFull, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) warp_sums[lane] = w;  // inclusive
    }
    __syncthreads();
    T warp_prefix = warp == 0 ? T(0) : warp_sums[warp - 1];
    if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
    T res = warp_prefix + x - v;
    __syncthreads();
    return res;
}

template <class T>
__device__ __forceinline__ void load_scan_items(const T* in, int64_t base, int64_t n, T* v) {
#pragma unroll
    for (int i = 0; i < kScanIPT; ++i) v[i] = (base + i < n) ? in[base + i] : T(0);
}
template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const T* in, T* sums, int64_t n) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanIPT;
    T v[kScanIPT], s = 0;
    load_scan_items(in, base, n, v);
#pragma unroll
    for (int i = 0; i < kScanIPT; ++i) s += v[i];
    T tot = 0;
    block_exclusive_scan<T>(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}
// The tile's items after the sums of the tiles before it (added up by every
// block in the same order), or after before[blockIdx.x] where that is given.
template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_tile_kernel(const T* in, T* out,
                                                                 const T* sums, const T* before,
                                                                 T* total, int64_t n) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanIPT;
    T v[kScanIPT], s = 0;
    T first = 0;
    if (before) {
        first = before[blockIdx.x];
    } else if (blockIdx.x > 0) {
        const int per = (int)((blockIdx.x + kScanThreads - 1) / kScanThreads);
        const int b0 = (int)threadIdx.x * per;
        T x = 0;
        for (int b = b0; b < b0 + per && b < (int)blockIdx.x; ++b) x += sums[b];
        block_exclusive_scan<T>(x, &first);
    }
    load_scan_items(in, base, n, v);
#pragma unroll
    for (int i = 0; i < kScanIPT; ++i) s += v[i];
    T tot = 0;
    T run = block_exclusive_scan<T>(s, &tot);
#pragma unroll
    for (int i = 0; i < kScanIPT; ++i) {
        if (base + i < n) out[base + i] = run + first;
        run += v[i];
    }
    if (threadIdx.x == 0 && total && blockIdx.x == gridDim.x - 1) *total = first + tot;
}

// Beyond this many tiles the tile sums are scanned themselves, as they always
// are for float64 (the order of whose additions is the result); up to it every
// block adds up those before it, a few words a thread.
constexpr int64_t kScanDirect = 4096;

template <class T>
int scan_exclusive(Workspace& ws, const T* in, T* out, int64_t n, T* total) {
    cudaStream_t s = ws.stream();
    if (n <= 0) {
        if (total) FHG_CUDA(cudaMemsetAsync(total, 0, sizeof(T), s));
        return FHG_OK;
    }
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    Workspace tmp(ws);
    T *sums = nullptr, *before = nullptr;
    if (tiles > 1) {
        FHG_TRY(tmp.alloc(&sums, (size_t)tiles));
        ::fhg::note_launch();
        scan_sums_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, sums, n);
        FHG_CUDA(cudaGetLastError());
        if (tiles > kScanDirect || std::is_same<T, double>::value) {
            FHG_TRY(tmp.alloc(&before, (size_t)tiles));
            FHG_TRY(scan_exclusive<T>(tmp, sums, before, tiles, nullptr));
        }
    }
    ::fhg::note_launch();
    scan_tile_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, sums, before, total, n);
    FHG_CUDA(cudaGetLastError());
    return FHG_OK;
}

// ---------------------------------------------------------------- radix sort
constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsSmall = 2048;  // items that one block sorts alone
constexpr int kRsMaxPasses = 8;
// 32-item rows of a warp.  A tile is one block's latency, and every tile reads
// the words of those before it that run beside it: few items want small tiles
// (20k items, ten digits: 114 us at 8 rows, 140 at 12), many want few (16M
// items, four digits: 914 and 764 us).  At 12 a tile fits the static 48 KB.
constexpr int kRsRowsFew = 8, kRsRowsMany = 12;
constexpr int64_t kRsMany = 1 << 19;
template <int ROWS>
__host__ __device__ constexpr int rs_tile() { return kRsWarps * ROWS * 32; }

// Counts of every digit of all passes: hist[pass][256].
template <class K>
__global__ void __launch_bounds__(kRsThreads) rs_hist_kernel(const K* __restrict__ keys,
                                                             int64_t n, int shift, int passes,
                                                             uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kRsMaxPasses][256];
    for (int i = threadIdx.x; i < passes * 256; i += kRsThreads) (&h[0][0])[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t step = (int64_t)gridDim.x * kRsThreads;
    for (int64_t i = (int64_t)blockIdx.x * kRsThreads + threadIdx.x; i - lane < n; i += step) {
        const bool valid = i < n;
        const K k = valid ? keys[i] : K(0);
        const unsigned act = __ballot_sync(kFull, valid);
        for (int p = 0; p < passes; ++p) {
            const unsigned d = (unsigned)(k >> (shift + 8 * p)) & 255u;
            // the high digits of a row are often all the same: one addition
            const unsigned d0 = __shfl_sync(kFull, d, 0);
            if (__all_sync(kFull, !valid || d == d0)) {
                if (lane == 0) atomicAdd(&h[p][d0], (uint32_t)__popc(act));
            } else if (valid) {
                atomicAdd(&h[p][d], 1u);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += kRsThreads) {
        const uint32_t c = (&h[0][0])[i];
        if (c) atomicAdd(&hist[i], c);
    }
}

// A published word: the pass and kind above 56 bits of count, so that one
// zeroed array serves every pass.
__device__ __forceinline__ unsigned long long rs_word(int pass, int kind, uint64_t count) {
    return ((unsigned long long)(2 * pass + kind) << 56) | count;
}
constexpr int kRsOwn = 1, kRsUpTo = 2;         // the tile's own count; all up to it
constexpr int kRsWaitPolls = 1 << 20;          // some tenths of a second
constexpr int kRsWindow = 8;

// One stable pass.  Each warp ranks its rows in order (the lanes of equal
// digit by eight ballots, per-warp running counts); the tile's items are then
// laid out in digit order in shared memory and written so that consecutive
// threads store consecutive positions of one digit's run.  What bounds it is
// memory at the largest sizes and the launch at the smallest; against a
// histogram, a scan and a scatter kernel per pass it reads the keys once less
// and takes one launch instead of four.
template <class K, int kRows>
__global__ void __launch_bounds__(kRsThreads, kRows <= 8 ? 5 : 4) rs_pass_kernel(
    const K* __restrict__ kin, const int32_t* __restrict__ vin, K* __restrict__ kout,
    int32_t* __restrict__ vout, int64_t n, int shift, int pass, const uint32_t* __restrict__ hist,
    uint32_t* __restrict__ counter, unsigned long long* __restrict__ state) {
    constexpr int kTile = rs_tile<kRows>();
    __shared__ uint32_t wcnt[kRsWarps][256];
    __shared__ uint32_t tstart[256];
    __shared__ int64_t gbase[256];
    __shared__ K skey[kTile];
    __shared__ int32_t sval[kTile];
    __shared__ uint32_t s_tile;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
    for (int i = threadIdx.x; i < kRsWarps * 256; i += kRsThreads) (&wcnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int64_t tile0 = tile * kTile;
    const int64_t base = tile0 + (int64_t)w * (kRows * 32);
    K key[kRows];
    uint32_t pos[kRows];
#pragma unroll
    for (int c = 0; c < kRows; ++c) {
        const int64_t idx = base + c * 32 + lane;
        key[c] = idx < n ? kin[idx] : K(0);
    }
    // The first lane of every digit in a row adds the row's lanes to the warp's
    // count; the count it found is wanted only after all rows, so that their
    // additions (in row order) do not wait for one another.
    unsigned peers[kRows];
#pragma unroll
    for (int c = 0; c < kRows; ++c) {
        const bool valid = base + c * 32 + lane < n;
        const unsigned d = (unsigned)(key[c] >> shift) & 255u;
        unsigned m = __ballot_sync(kFull, valid);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const bool bit = (d >> b) & 1u;
            const unsigned on = __ballot_sync(kFull, bit);
            m &= bit ? on : ~on;
        }
        peers[c] = m;
        pos[c] = 0;
        if (valid && (m & lt_mask) == 0) pos[c] = atomicAdd(&wcnt[w][d], (uint32_t)__popc(m));
        __syncwarp();
    }
#pragma unroll
    for (int c = 0; c < kRows; ++c)
        pos[c] = __shfl_sync(kFull, pos[c], max(__ffs(peers[c]) - 1, 0)) +
                 __popc(peers[c] & lt_mask);
    int32_t val[kRows];  // (on their way while the block scans its counts)
#pragma unroll
    for (int c = 0; c < kRows; ++c) {
        const int64_t idx = base + c * 32 + lane;
        val[c] = idx < n ? vin[idx] : 0;
    }
    __syncthreads();
    const int d = threadIdx.x;  // this thread's digit
    uint32_t count = 0;
    for (int ww = 0; ww < kRsWarps; ++ww) {  // the warps' offsets inside the digit
        const uint32_t c = wcnt[ww][d];
        wcnt[ww][d] = count;
        count += c;
    }
    volatile unsigned long long* word = state + tile * 256 + d;
    *word = rs_word(pass, tile == 0 ? kRsUpTo : kRsOwn, count);
    tstart[d] = block_exclusive_scan<uint32_t>(count, nullptr);
    const uint32_t first = block_exclusive_scan<uint32_t>(hist[d], nullptr);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kRows; ++c) {
        if (base + c * 32 + lane < n) {
            const unsigned dg = (unsigned)(key[c] >> shift) & 255u;
            const uint32_t lp = tstart[dg] + wcnt[w][dg] + pos[c];
            skey[lp] = key[c];
            sval[lp] = val[c];
        }
    }
    // ---- the digit's items in the tiles before this one
    // (kRsWindow words at a time: tiles that run side by side have published
    // their own counts only, and a walk over them one by one is one read's
    // latency each)
    uint64_t before = 0;
    bool lost = false, done = tile == 0;
    int polls = 0;
    for (int64_t t = tile - 1; !done;) {
        unsigned long long x[kRsWindow];
#pragma unroll
        for (int j = 0; j < kRsWindow; ++j)
            x[j] = t - j >= 0 ? *(const volatile unsigned long long*)(state + (t - j) * 256 + d)
                              : 0ull;
        int taken = 0;
#pragma unroll
        for (int j = 0; j < kRsWindow; ++j) {
            // in order, up to one not published in this pass yet
            if (!done && taken == j && (int)(x[j] >> 56) > 2 * pass) {
                before += x[j] & ((1ull << 56) - 1ull);
                done = (int)(x[j] >> 56) == 2 * pass + kRsUpTo;
                ++taken;
            }
        }
        t -= taken;
        if (!done && taken == 0) {
            if (++polls > kRsWaitPolls) {
                lost = true;
                break;
            }
            if (polls > 16) __nanosleep(64);
        }
    }
    if (__syncthreads_or(lost)) {  // count them from the keys
        wcnt[0][d] = 0;
        __syncthreads();
        for (int64_t i = threadIdx.x; i < tile0; i += kRsThreads)
            atomicAdd(&wcnt[0][(unsigned)(kin[i] >> shift) & 255u], 1u);
        __syncthreads();
        before = wcnt[0][d];
    }
    if (tile > 0) *word = rs_word(pass, kRsUpTo, before + count);
    gbase[d] = (int64_t)(first + before) - (int64_t)tstart[d];
    __syncthreads();
    const int cnt = (int)(n - tile0 < kTile ? n - tile0 : kTile);
    for (int i = threadIdx.x; i < cnt; i += kRsThreads) {
        const K k = skey[i];
        const int64_t dst = gbase[(unsigned)(k >> shift) & 255u] + i;
        kout[dst] = k;
        vout[dst] = sval[i];
    }
}

// The same sort for n <= kRsSmall in one launch: a bitonic sort in shared
// memory of (digits, position) pairs, where digits are the key bits the LSD
// passes cover ([begin, end) rounded up to whole 8-bit digits), so the order
// is the stable one the passes give.
constexpr int kRsSmallThreads = 1024;
template <class K>
__global__ void __launch_bounds__(kRsSmallThreads) rs_small_kernel(K* keys, int32_t* vals, int n,
                                                                   int shift, int bits) {
    __shared__ K sk[kRsSmall];
    __shared__ uint16_t si[kRsSmall];
    __shared__ int32_t sv[kRsSmall];
    const K mask = bits >= (int)(8 * sizeof(K)) ? ~K(0) : ((K(1) << bits) - K(1));
    int m2 = 1;
    while (m2 < n) m2 <<= 1;
    for (int i = threadIdx.x; i < m2; i += blockDim.x) {
        sk[i] = i < n ? keys[i] : ~K(0);
        si[i] = i < n ? (uint16_t)i : (uint16_t)0xffffu;  // padding sorts last
        if (i < n) sv[i] = vals ? vals[i] : 0;
    }
    __syncthreads();
    for (int size = 2; size <= m2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < m2; i += blockDim.x) {
                const int j = i ^ stride;
                if (j > i) {
                    const K da = (sk[i] >> shift) & mask, db = (sk[j] >> shift) & mask;
                    const bool greater = da > db || (da == db && si[i] > si[j]);
                    if (greater == ((i & size) == 0)) {
                        const K tk = sk[i];
                        sk[i] = sk[j];
                        sk[j] = tk;
                        const uint16_t ti = si[i];
                        si[i] = si[j];
                        si[j] = ti;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        keys[i] = sk[i];
        if (vals) vals[i] = sv[si[i]];
    }
}

template <class K>
int radix_sort(Workspace& ws, K* keys, int32_t* vals, int64_t n, int begin_bit, int end_bit) {
    if (n <= 1 || end_bit <= begin_bit) return FHG_OK;
    if (n >= ((int64_t)1 << 32)) {
        set_error("radix sort: n too large");
        return FHG_ERR_INVALID;
    }
    cudaStream_t s = ws.stream();
    if (n <= kRsSmall) {
        const int bits = std::min(((end_bit - begin_bit + 7) / 8) * 8,
                                  (int)(8 * sizeof(K)) - begin_bit);
        ::fhg::note_launch();
        rs_small_kernel<K><<<1, kRsSmallThreads, 0, s>>>(keys, vals, (int)n, begin_bit, bits);
        FHG_CUDA(cudaGetLastError());
        return FHG_OK;
    }
    const int passes = (end_bit - begin_bit + 7) / 8;
    const bool many = n > kRsMany;
    const int tile = many ? rs_tile<kRsRowsMany>() : rs_tile<kRsRowsFew>();
    const int64_t tiles = (n + tile - 1) / tile;
    Workspace tmp(ws);
    // an odd number of passes over two buffers would end in the other one
    K* kb[3] = {keys, nullptr, nullptr};
    int32_t* vb[3] = {vals, nullptr, nullptr};
    const int spare = passes >= 3 && (passes & 1) ? 2 : 1;
    for (int i = 1; i <= spare; ++i) {
        FHG_TRY(tmp.alloc(&kb[i], (size_t)n));
        FHG_TRY(tmp.alloc(&vb[i], (size_t)n));
    }
    // [tile counters][digit counts][published words], zeroed together
    constexpr size_t kHead = kRsMaxPasses + kRsMaxPasses * 256;
    uint32_t* head;
    const size_t words = kHead + 2 * (size_t)tiles * 256;
    FHG_TRY(tmp.alloc(&head, words));
    unsigned long long* state = reinterpret_cast<unsigned long long*>(head + kHead);
    FHG_CUDA(cudaMemsetAsync(head, 0, words * sizeof(uint32_t), s));
    ::fhg::note_launch();
    rs_hist_kernel<K><<<(unsigned)std::min<int64_t>((n + 1023) / 1024, 6 * 152), kRsThreads, 0,
                        s>>>(
        keys, n, begin_bit, passes, head + kRsMaxPasses);
    FHG_CUDA(cudaGetLastError());
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        const int to = p + 1 == passes && passes > 1 ? 0 : (cur == 1 ? (spare == 2 ? 2 : 0) : 1);
        ::fhg::note_launch();
        const auto pass = many ? rs_pass_kernel<K, kRsRowsMany> : rs_pass_kernel<K, kRsRowsFew>;
        pass<<<(unsigned)tiles, kRsThreads, 0, s>>>(
            kb[cur], vb[cur], kb[to], vb[to], n, begin_bit + 8 * p, p,
            head + kRsMaxPasses + 256 * p, head + p, state);
        FHG_CUDA(cudaGetLastError());
        cur = to;
    }
    if (cur != 0) {
        FHG_CUDA(cudaMemcpyAsync(keys, kb[cur], sizeof(K) * n, cudaMemcpyDeviceToDevice, s));
        FHG_CUDA(cudaMemcpyAsync(vals, vb[cur], sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s));
    }
    return FHG_OK;
}

__global__ void iota_kernel(int32_t* p, int64_t n) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = (int32_t)i;
}

}  // namespace

int scan_exclusive_u32(Workspace& ws, const uint32_t* in, uint32_t* out, int64_t n,
                       uint32_t* total) {
    return scan_exclusive<uint32_t>(ws, in, out, n, total);
}
int scan_exclusive_i64(Workspace& ws, const int64_t* in, int64_t* out, int64_t n,
                       int64_t* total) {
    return scan_exclusive<int64_t>(ws, in, out, n, total);
}
int scan_exclusive_f64(Workspace& ws, const double* in, double* out, int64_t n, double* total) {
    return scan_exclusive<double>(ws, in, out, n, total);
}
int radix_sort_u64(Workspace& ws, uint64_t* keys, int32_t* vals, int64_t n, int begin_bit,
                   int end_bit) {
    return radix_sort<uint64_t>(ws, keys, vals, n, begin_bit, end_bit);
}
int radix_sort_u32(Workspace& ws, uint32_t* keys, int32_t* vals, int64_t n, int begin_bit,
                   int end_bit) {
    return radix_sort<uint32_t>(ws, keys, vals, n, begin_bit, end_bit);
}
int fill_iota_i32(int32_t* p, int64_t n, cudaStream_t s) {
    if (n <= 0) return FHG_OK;
    ::fhg::note_launch();
    iota_kernel<<<grid_for(n, 256), 256, 0, s>>>(p, n);
    FHG_CUDA(cudaGetLastError());
    return FHG_OK;
}

}  // namespace fhg
