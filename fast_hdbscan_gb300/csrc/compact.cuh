// Stable stream compaction in two launches (one for up to kCompactOne
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

// A thread's indices, THREADS apart.  A tile of 256 x 16 reads its counts least
// often; but test and emit are chains of gathers, and below kCompactFew indices
// (two rounds of blocks) its few blocks are latency: there a thread takes 2 (200k
// components, the round's edges: 182 -> 32 us).  One block takes what fits in it.
constexpr int kCompactThreads = 256, kCompactRows = 16, kCompactFewRows = 2;
constexpr int kCompactOneThreads = 1024, kCompactOneRows = 4;
constexpr int64_t kCompactFew = (int64_t)2 * 152 * kCompactThreads * kCompactRows;
constexpr int64_t kCompactOne = kCompactOneThreads * kCompactOneRows;
constexpr int64_t kCompactScan = 2048;

template <class F, int THREADS, int ROWS>
__global__ void __launch_bounds__(THREADS) compact_count_kernel(F f, int64_t n,
                                                                uint32_t* counts) {
    const int64_t base = (int64_t)blockIdx.x * (THREADS * ROWS) + threadIdx.x;
    int c = 0;
#pragma unroll
    for (int t = 0; t < ROWS; ++t) {
        const int64_t i = base + t * THREADS;
        c += i < n && f.test(i) ? 1 : 0;
    }
    __shared__ int s_c[THREADS / 32];
    c = __reduce_add_sync(kFull, c);
    if ((threadIdx.x & 31) == 0) s_c[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int sum = 0;
        for (int w = 0; w < THREADS / 32; ++w) sum += s_c[w];
        counts[blockIdx.x] = (uint32_t)sum;
    }
}

template <class F, int THREADS, int ROWS>
__global__ void __launch_bounds__(THREADS) compact_emit_kernel(F f, int64_t n,
                                                               const uint32_t* counts,
                                                               bool scanned, uint32_t* total) {
    constexpr int kWarps = THREADS / 32;
    __shared__ uint32_t s_cell[ROWS][kWarps];  // marked indices per row and warp
    __shared__ uint32_t s_before;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_before = 0;
    __syncthreads();
    uint32_t before = 0;
    if (scanned) {
        before = threadIdx.x == 0 ? counts[blockIdx.x] : 0u;
    } else {
        for (int64_t b = threadIdx.x; b < (int64_t)blockIdx.x; b += THREADS)
            before += counts[b];
    }
    before = __reduce_add_sync(kFull, before);
    if (lane == 0 && before) atomicAdd(&s_before, before);
    const int64_t base = (int64_t)blockIdx.x * (THREADS * ROWS) + threadIdx.x;
    unsigned mine[ROWS];
#pragma unroll
    for (int t = 0; t < ROWS; ++t) {
        const int64_t i = base + t * THREADS;
        mine[t] = __ballot_sync(kFull, i < n && f.test(i));
        if (lane == 0) s_cell[t][w] = __popc(mine[t]);
    }
    __syncthreads();
    if (w == 0) {  // exclusive prefix of the cells, in index order
        constexpr int kCells = ROWS * kWarps, kPer = (kCells + 31) / 32;
        uint32_t v[kPer], sum = 0;
        uint32_t* cell = &s_cell[0][0] + lane * kPer;
        const bool mine_too = lane * kPer < kCells;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            v[j] = mine_too ? cell[j] : 0u;
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
            if (mine_too) cell[j] = run;
            run += v[j];
        }
        if (lane == 31 && total && blockIdx.x == gridDim.x - 1) *total = run;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < ROWS; ++t) {
        const int64_t i = base + t * THREADS;
        if (i >= n) break;
        f.each(i);
        if ((mine[t] >> lane) & 1u)
            f.emit(i, s_cell[t][w] + __popc(mine[t] & ((1u << lane) - 1u)));
    }
}

template <class F, int THREADS, int ROWS>
int compact_tiles(Workspace& ws, const F& f, int64_t n, uint32_t* total) {
    static_assert(ROWS * THREADS / 32 <= 32 || ROWS * THREADS / 32 % 32 == 0, "whole lanes");
    cudaStream_t s = ws.stream();
    const int64_t tiles = (n + THREADS * ROWS - 1) / (THREADS * ROWS);
    Workspace tmp(ws);
    uint32_t *counts = nullptr, *starts = nullptr;
    const bool scanned = tiles > kCompactScan;
    if (tiles > 1) {
        FHG_TRY(tmp.alloc(&counts, (size_t)tiles));
        if (scanned) FHG_TRY(tmp.alloc(&starts, (size_t)tiles));
        ::fhg::note_launch();
        compact_count_kernel<F, THREADS, ROWS><<<(unsigned)tiles, THREADS, 0, s>>>(f, n, counts);
        FHG_CUDA(cudaGetLastError());
        if (scanned) FHG_TRY(scan_exclusive_u32(tmp, counts, starts, tiles, nullptr));
    }
    ::fhg::note_launch();
    compact_emit_kernel<F, THREADS, ROWS><<<(unsigned)tiles, THREADS, 0, s>>>(
        f, n, scanned ? starts : counts, scanned, total);
    FHG_CUDA(cudaGetLastError());
    return FHG_OK;
}

// total (device, nullable) receives the number of marked indices.
template <class F>
int compact(Workspace& ws, const F& f, int64_t n, uint32_t* total) {
    if (n <= 0) {
        if (total) FHG_CUDA(cudaMemsetAsync(total, 0, sizeof(uint32_t), ws.stream()));
        return FHG_OK;
    }
    if (n <= kCompactOne)
        return compact_tiles<F, kCompactOneThreads, kCompactOneRows>(ws, f, n, total);
    if (n < kCompactFew)
        return compact_tiles<F, kCompactThreads, kCompactFewRows>(ws, f, n, total);
    return compact_tiles<F, kCompactThreads, kCompactRows>(ws, f, n, total);
}

}  // namespace fhg
