// Stable stream compaction in two launches (one for up to kCompactTile
// indices): the indices i of [0, n) with f.test(i), in order, get the places
// 0, 1, ... by f.emit(i, place).
//
// F is a struct of device pointers with
//   __device__ bool test(int64_t i) const;
//   __device__ void emit(int64_t i, uint32_t place) const;  // tested ones
//   __device__ void each(int64_t i) const;                  // every index
// test may not read what emit or each writes.  The first launch counts every
// tile; in the second each block adds up the counts of the tiles before its
// own (at most a few thousand words, from L2) and places its indices.  Against
// flags, a three-launch scan of them and a gather this halves the launches and
// leaves out two passes over n words.  Past kCompactScan tiles (8M indices) the
// blocks' sums grow to a good part of what the indices themselves take (their
// reads with the square of n), and a scan of the counts takes their place.
#pragma once
#include "fhg_common.cuh"
#include "primitives.cuh"

namespace fhg {

constexpr int kCompactThreads = 256;
constexpr int kCompactRows = 16;  // indices of a thread, kCompactThreads apart
constexpr int kCompactTile = kCompactThreads * kCompactRows;
constexpr int64_t kCompactScan = 2048;

template <class F>
__global__ void __launch_bounds__(kCompactThreads) compact_count_kernel(F f, int64_t n,
                                                                        uint32_t* counts) {
    const int64_t base = (int64_t)blockIdx.x * kCompactTile + threadIdx.x;
    int c = 0;
#pragma unroll
    for (int t = 0; t < kCompactRows; ++t) {
        const int64_t i = base + t * kCompactThreads;
        c += i < n && f.test(i) ? 1 : 0;
    }
    __shared__ int s_c[kCompactThreads / 32];
    c = __reduce_add_sync(kFull, c);
    if ((threadIdx.x & 31) == 0) s_c[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int sum = 0;
        for (int w = 0; w < kCompactThreads / 32; ++w) sum += s_c[w];
        counts[blockIdx.x] = (uint32_t)sum;
    }
}

template <class F>
__global__ void __launch_bounds__(kCompactThreads) compact_emit_kernel(F f, int64_t n,
                                                                       const uint32_t* counts,
                                                                       bool scanned,
                                                                       uint32_t* total) {
    constexpr int kWarps = kCompactThreads / 32;
    __shared__ uint32_t s_cell[kCompactRows][kWarps];  // marked indices per row and warp
    __shared__ uint32_t s_before;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_before = 0;
    __syncthreads();
    uint32_t before = 0;
    if (scanned) {
        before = threadIdx.x == 0 ? counts[blockIdx.x] : 0u;
    } else {
        for (int64_t b = threadIdx.x; b < (int64_t)blockIdx.x; b += kCompactThreads)
            before += counts[b];
    }
    before = __reduce_add_sync(kFull, before);
    if (lane == 0 && before) atomicAdd(&s_before, before);
    const int64_t base = (int64_t)blockIdx.x * kCompactTile + threadIdx.x;
    unsigned mine[kCompactRows];
#pragma unroll
    for (int t = 0; t < kCompactRows; ++t) {
        const int64_t i = base + t * kCompactThreads;
        mine[t] = __ballot_sync(kFull, i < n && f.test(i));
        if (lane == 0) s_cell[t][w] = __popc(mine[t]);
    }
    __syncthreads();
    if (w == 0) {  // exclusive prefix of the cells, in index order
        constexpr int kCells = kCompactRows * kWarps, kPer = kCells / 32;
        uint32_t v[kPer], sum = 0;
        uint32_t* cell = &s_cell[0][0] + lane * kPer;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            v[j] = cell[j];
            sum += v[j];
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        uint32_t run = s_before + x - sum;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            cell[j] = run;
            run += v[j];
        }
        if (lane == 31 && total && blockIdx.x == gridDim.x - 1) *total = run;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kCompactRows; ++t) {
        const int64_t i = base + t * kCompactThreads;
        if (i >= n) break;
        f.each(i);
        if ((mine[t] >> lane) & 1u)
            f.emit(i, s_cell[t][w] + __popc(mine[t] & ((1u << lane) - 1u)));
    }
}

// total (device, nullable) receives the number of marked indices.
template <class F>
int compact(Workspace& ws, const F& f, int64_t n, uint32_t* total) {
    cudaStream_t s = ws.stream();
    if (n <= 0) {
        if (total) FHG_CUDA(cudaMemsetAsync(total, 0, sizeof(uint32_t), s));
        return FHG_OK;
    }
    const int64_t tiles = (n + kCompactTile - 1) / kCompactTile;
    Workspace tmp(ws);
    uint32_t *counts = nullptr, *starts = nullptr;
    const bool scanned = tiles > kCompactScan;
    if (tiles > 1) {
        FHG_TRY(tmp.alloc(&counts, (size_t)tiles));
        if (scanned) FHG_TRY(tmp.alloc(&starts, (size_t)tiles));
        ::fhg::note_launch();
        compact_count_kernel<F><<<(unsigned)tiles, kCompactThreads, 0, s>>>(f, n, counts);
        FHG_CUDA(cudaGetLastError());
        if (scanned) FHG_TRY(scan_exclusive_u32(tmp, counts, starts, tiles, nullptr));
    }
    ::fhg::note_launch();
    compact_emit_kernel<F><<<(unsigned)tiles, kCompactThreads, 0, s>>>(f, n, scanned ? starts : counts,
                                                                     scanned, total);
    FHG_CUDA(cudaGetLastError());
    return FHG_OK;
}

}  // namespace fhg
