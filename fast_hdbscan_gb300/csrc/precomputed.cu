// Precomputed sparse graphs (metric="precomputed"): precomputed.py:479
// compute_mst_from_precomputed_sparse_kruskal and :410
// compute_mst_from_precomputed_sparse, without cannot-link constraints.
//
// The reference symmetrises the graph by the least weight per undirected pair
// without its diagonal (:70 _symmetrize_min_csr), takes every point's core
// distance as the min_samples-th smallest weight of its row (:148
// _core_distances_csr), gives every stored entry its float64
// mutual-reachability weight max(core_i, core_j, w_ij) and builds the minimum
// spanning forest -- Kruskal over a stable argsort of the entries, or its
// float32 Boruvka -- then joins the components with +inf bridges.
//
// Here: the least weight of every pair by a stable radix sort of the (min, max)
// pair keys with a segmented minimum.  A row of the symmetric matrix is then its
// pairs (i, j) with i < j, which stand together in pair order, and the mirrored
// ones, stably by row, as the reference's two concatenated halves: only these
// are sorted.  A warp per row ranks its entries by (weight, position) for the
// core distance and the neighbours.  A pair's two entries have one weight and
// the one with i < j comes first, so the other is never accepted: the pairs
// alone are sorted by weight, and the forest comes from the Boruvka rounds over
// sorted ranks of kruskal.cu.  The forest is Kruskal's (float64 weight, then
// entry position) for both algorithms: the reference's Boruvka returns a forest
// of the same weights, whose equal-weight choices and edge order are its own.
//
// What bounds it is the sorts' digit passes: 5 over the entries and 3 + 8 over
// the pairs (before: 5, and 3 + 8 + 3 + 8 over both entries of every pair).
// 300k rows, 15 neighbours each: 4.5 -> 1.9 ms with the forest.
#include "mst.cuh"
#include "primitives.cuh"

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

__device__ __forceinline__ uint64_t f64_bits(double x) {  // x >= 0 (or +inf)
    return (uint64_t)__double_as_longlong(x);
}

__global__ void pc_offdiag_kernel(int64_t nnz, const int32_t* __restrict__ rows,
                                  const int32_t* __restrict__ cols, uint32_t* __restrict__ flag) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nnz) flag[t] = rows[t] != cols[t] ? 1u : 0u;
}
// (min, max) pair key of every off-diagonal entry, in input order, and its
// weight, with -0.0 as 0.0: from here on weights are ordered by their bits, and
// the forest's edges are taken to come in ascending order.
__global__ void pc_pairs_kernel(int64_t nnz, int64_t n, const int32_t* __restrict__ rows,
                                const int32_t* __restrict__ cols, const double* __restrict__ data,
                                const uint32_t* __restrict__ flag, const uint32_t* __restrict__ pos,
                                uint64_t* __restrict__ key, int32_t* __restrict__ at,
                                double* __restrict__ d0) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nnz || !flag[t]) return;
    const int64_t u = min(rows[t], cols[t]), v = max(rows[t], cols[t]);
    const uint32_t o = pos[t];
    key[o] = (uint64_t)u * (uint64_t)n + (uint64_t)v;
    at[o] = (int32_t)o;
    d0[o] = data[t] + 0.0;
}
__global__ void pc_group_flags_kernel(int64_t m0, const uint64_t* __restrict__ key,
                                      uint32_t* __restrict__ flag) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < m0) flag[j] = (j == 0 || key[j] != key[j - 1]) ? 1u : 0u;
}
__global__ void pc_fill_u64_kernel(uint64_t* a, int64_t n, uint64_t v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = v;
}
// np.minimum.reduceat over each pair's run (the weights are >= 0, so their
// bit patterns order like the values).
__global__ void pc_group_min_kernel(int64_t m0, int64_t n, const uint64_t* __restrict__ key,
                                    const int32_t* __restrict__ at, const double* __restrict__ d0,
                                    const uint32_t* __restrict__ flag,
                                    const uint32_t* __restrict__ gpos,
                                    unsigned long long* __restrict__ gmin,
                                    int32_t* __restrict__ gu, int32_t* __restrict__ gv) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m0) return;
    // group of j: the last group start at or before j
    const int64_t g = (int64_t)gpos[j] + (flag[j] ? 0 : -1);
    atomicMin(&gmin[g], (unsigned long long)f64_bits(d0[at[j]]));
    if (flag[j]) {
        gu[g] = (int32_t)(key[j] / (uint64_t)n);
        gv[g] = (int32_t)(key[j] % (uint64_t)n);
    }
}
// The mirrored entries (v, u), in pair order.
__global__ void pc_mirror_kernel(int64_t mu, const int32_t* __restrict__ gv,
                                 uint32_t* __restrict__ rowkey, int32_t* __restrict__ perm) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= mu) return;
    rowkey[t] = (uint32_t)gv[t];
    perm[t] = (int32_t)t;
}
template <class T>
__device__ __forceinline__ int64_t pc_lower_bound(const T* __restrict__ a, int64_t n, T v) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
// Where row r's pairs (among gu) and mirrored entries (among the sorted vrow)
// start, r in [0, n]; longest = the longest row.
__global__ void pc_rows_kernel(int64_t n, int64_t mu, const int32_t* __restrict__ gu,
                               const uint32_t* __restrict__ vrow, uint32_t* __restrict__ ubeg,
                               uint32_t* __restrict__ lbeg, uint32_t* __restrict__ longest) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t len = 0;
    if (r <= n) {
        const int64_t u = pc_lower_bound(gu, mu, (int32_t)r);
        const int64_t l = pc_lower_bound(vrow, mu, (uint32_t)r);
        ubeg[r] = (uint32_t)u;
        lbeg[r] = (uint32_t)l;
        if (r < n)
            len = (uint32_t)(pc_lower_bound(gu, mu, (int32_t)r + 1) - u +
                             pc_lower_bound(vrow, mu, (uint32_t)r + 1) - l);
    }
    len = __reduce_max_sync(kFull, len);
    if ((threadIdx.x & 31) == 0 && len > *(volatile uint32_t*)longest) atomicMax(longest, len);
}
// :148 _core_distances_csr, a warp per row of up to kPcRow entries: an entry's
// place is the number of entries of the row before it in (weight, position).
// Longer rows are ordered by sorting all entries by weight and by row, eleven
// digit passes however long the rows; ranking takes len^2 / 32 steps a row (4M
// entries, rows of 16 / 64 / 256: 1.40 / 1.29 / 1.54 ms for the whole tree, by
// sorting 2.26 / 2.07 / 2.24).
constexpr int kPcRow = 256, kPcWarps = 4;
__global__ void __launch_bounds__(kPcWarps * 32) pc_rank_rows_kernel(
    int64_t n, int k, int ms, const int32_t* __restrict__ gu, const int32_t* __restrict__ gv,
    const unsigned long long* __restrict__ gmin, const int32_t* __restrict__ lperm,
    const uint32_t* __restrict__ ubeg, const uint32_t* __restrict__ lbeg,
    int32_t* __restrict__ nbrs, double* __restrict__ core) {
    __shared__ unsigned long long s_w[kPcWarps][kPcRow];
    __shared__ int32_t s_col[kPcWarps][kPcRow];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t r = (int64_t)blockIdx.x * kPcWarps + warp;
    if (r >= n) return;
    const uint32_t u0 = ubeg[r], l0 = lbeg[r];
    const int nu = (int)(ubeg[r + 1] - u0), len = nu + (int)(lbeg[r + 1] - l0);
    for (int e = lane; e < len; e += 32) {
        const int64_t g = e < nu ? u0 + e : lperm[l0 + (e - nu)];
        s_w[warp][e] = gmin[g];
        s_col[warp][e] = e < nu ? gv[g] : gu[g];
    }
    __syncwarp();
    for (int e = lane; e < len; e += 32) {
        const unsigned long long w = s_w[warp][e];
        int at = 0;
        for (int o = 0; o < len; ++o) {
            const unsigned long long x = s_w[warp][o];
            at += x < w || (x == w && o < e) ? 1 : 0;
        }
        if (at < k) nbrs[r * k + at] = s_col[warp][e];
        if (ms > 1 && at == ms - 1) core[r] = __longlong_as_double((long long)w);
    }
}
// Both halves one behind the other, for rows too long to rank.
__global__ void pc_sym_kernel(int64_t mu, const int32_t* __restrict__ gu,
                              const int32_t* __restrict__ gv, uint32_t* __restrict__ rowkey,
                              int32_t* __restrict__ perm) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * mu) return;
    rowkey[t] = (uint32_t)(t < mu ? gu[t] : gv[t - mu]);
    perm[t] = (int32_t)t;
}
__global__ void pc_csr_kernel(int64_t M, int64_t mu, const int32_t* __restrict__ perm,
                              const int32_t* __restrict__ gu, const int32_t* __restrict__ gv,
                              const unsigned long long* __restrict__ gmin,
                              int32_t* __restrict__ srow, int32_t* __restrict__ scol,
                              double* __restrict__ sd, uint32_t* __restrict__ count) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= M) return;
    const int64_t t = perm[p];
    const int64_t g = t < mu ? t : t - mu;
    const int32_t r = t < mu ? gu[g] : gv[g];
    srow[p] = r;
    scol[p] = t < mu ? gv[g] : gu[g];
    sd[p] = __longlong_as_double((long long)gmin[g]);
    atomicAdd(&count[r], 1u);
}
__global__ void pc_weight_keys_kernel(int64_t M, const double* __restrict__ sd,
                                      uint64_t* __restrict__ key, int32_t* __restrict__ perm) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= M) return;
    key[p] = f64_bits(sd[p]);
    perm[p] = (int32_t)p;
}
__global__ void pc_row_keys_kernel(int64_t M, const int32_t* __restrict__ perm,
                                   const int32_t* __restrict__ srow, uint32_t* __restrict__ key) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < M) key[q] = (uint32_t)srow[perm[q]];
}
__global__ void pc_core_init_kernel(int64_t n, int k, int ms, int32_t* __restrict__ nbrs,
                                    double* __restrict__ core) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n * k) nbrs[t] = -1;
    if (t < n) core[t] = ms > 1 ? INFINITY : 0.0;
}
// :148 _core_distances_csr on the rows ordered by weight (ties by position).
__global__ void pc_core_kernel(int64_t M, int k, int ms, const int32_t* __restrict__ perm,
                               const int32_t* __restrict__ srow, const int32_t* __restrict__ scol,
                               const double* __restrict__ sd, const uint32_t* __restrict__ indptr,
                               int32_t* __restrict__ nbrs, double* __restrict__ core) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= M) return;
    const int32_t p = perm[q];
    const int32_t r = srow[p];
    const int64_t j = q - (int64_t)indptr[r];
    if (j < k) nbrs[(int64_t)r * k + j] = scol[p];
    if (ms > 1 && j == ms - 1) core[r] = sd[p];
}
// kruskal.py:421 _compute_mrd_csr_flat, of every pair's first entry.
__global__ void pc_mrd_kernel(int64_t mu, const int32_t* __restrict__ gu,
                              const int32_t* __restrict__ gv,
                              const unsigned long long* __restrict__ gmin,
                              const double* __restrict__ core, uint64_t* __restrict__ key,
                              int32_t* __restrict__ perm) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= mu) return;
    double mrd = core[gu[g]];
    const double cj = core[gv[g]], d = __longlong_as_double((long long)gmin[g]);
    if (cj > mrd) mrd = cj;
    if (d > mrd) mrd = d;
    key[g] = f64_bits(mrd);
    perm[g] = (int32_t)g;
}
__global__ void pc_ranks_kernel(int64_t mu, const int32_t* __restrict__ perm,
                                const int32_t* __restrict__ gu, const int32_t* __restrict__ gv,
                                int2* __restrict__ uv) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= mu) return;
    const int32_t g = perm[r];
    uv[r] = make_int2(gu[g], gv[g]);
}

// _core_distances_csr by sorting: the symmetric CSR, every row by weight, ties
// by position.
int core_by_sorting(Workspace& outer, int64_t n, int64_t mu, int k, int ms, const int32_t* gu,
                    const int32_t* gv, const unsigned long long* gmin, int32_t* neighbors,
                    double* core) {
    cudaStream_t s = outer.stream();
    Workspace ws(outer);
    const int64_t M = 2 * mu;
    uint32_t *rowkey, *count, *indptr;
    int32_t *perm, *srow, *scol;
    double* sd;
    uint64_t* wkey;
    FHG_TRY(ws.alloc(&rowkey, (size_t)M));
    FHG_TRY(ws.alloc(&perm, (size_t)M));
    FHG_TRY(ws.alloc(&srow, (size_t)M));
    FHG_TRY(ws.alloc(&scol, (size_t)M));
    FHG_TRY(ws.alloc(&sd, (size_t)M));
    FHG_TRY(ws.alloc(&count, (size_t)n));
    FHG_TRY(ws.alloc(&indptr, (size_t)n));
    FHG_TRY(ws.alloc(&wkey, (size_t)M));
    FHG_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t) * n, s));
    LAUNCH(pc_sym_kernel, M, mu, gu, gv, rowkey, perm);
    {
        Workspace tmp(ws);
        FHG_TRY(radix_sort_u32(tmp, rowkey, perm, M, 0, bits_for(n)));
    }
    LAUNCH(pc_csr_kernel, M, M, mu, perm, gu, gv, gmin, srow, scol, sd, count);
    FHG_TRY(scan_exclusive_u32(ws, count, indptr, n, nullptr));
    LAUNCH(pc_weight_keys_kernel, M, M, sd, wkey, perm);
    {
        Workspace tmp(ws);
        FHG_TRY(radix_sort_u64(tmp, wkey, perm, M, 0, 64));
    }
    LAUNCH(pc_row_keys_kernel, M, M, perm, srow, rowkey);
    {
        Workspace tmp(ws);
        FHG_TRY(radix_sort_u32(tmp, rowkey, perm, M, 0, bits_for(n)));
    }
    LAUNCH(pc_core_kernel, M, M, k, ms, perm, srow, scol, sd, indptr, neighbors, core);
    return FHG_OK;
}

}  // namespace

int precomputed_mst(const int32_t* rows, const int32_t* cols, const double* data, int64_t nnz,
                    int64_t n, int min_samples, double* edges, int32_t* neighbors, double* core,
                    int64_t* n_components, cudaStream_t s) {
    if (nnz > 0x7fffffffLL) {
        set_error("precomputed: %lld stored entries exceed the int32 entry index",
                  (long long)nnz);
        return FHG_ERR_UNSUPPORTED;
    }
    const int k = min_samples > 1 ? min_samples : 1;
    *n_components = n > 0 ? 1 : 0;
    if (n < 1) return FHG_OK;
    Stage stage(s, "precomputed_mst");
    Workspace ws(s);
    uint32_t* cnt;
    FHG_TRY(ws.alloc(&cnt, 2));
    LAUNCH(pc_core_init_kernel, n * k, n, k, min_samples, neighbors, core);

    // ---- _symmetrize_min_csr
    const size_t nz = (size_t)(nnz > 0 ? nnz : 1);
    uint32_t *flag, *pos;
    FHG_TRY(ws.alloc(&flag, nz));
    FHG_TRY(ws.alloc(&pos, nz));
    LAUNCH(pc_offdiag_kernel, nnz, nnz, rows, cols, flag);
    FHG_TRY(scan_exclusive_u32(ws, flag, pos, nnz, cnt));
    uint32_t h = 0;
    FHG_CUDA(cudaMemcpyAsync(&h, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    const int64_t m0 = h;
    const size_t mz = (size_t)(m0 > 0 ? m0 : 1);
    uint64_t* key;
    int32_t* at;
    double* d0;
    FHG_TRY(ws.alloc(&key, mz));
    FHG_TRY(ws.alloc(&at, mz));
    FHG_TRY(ws.alloc(&d0, mz));
    LAUNCH(pc_pairs_kernel, nnz, nnz, n, rows, cols, data, flag, pos, key, at, d0);
    if (m0 > 1) {
        Workspace tmp(ws);
        const int kb = 2 * bits_for(n);
        FHG_TRY(radix_sort_u64(tmp, key, at, m0, 0, kb < 64 ? kb : 64));
    }
    uint32_t *gflag, *gpos;
    FHG_TRY(ws.alloc(&gflag, mz));
    FHG_TRY(ws.alloc(&gpos, mz));
    LAUNCH(pc_group_flags_kernel, m0, m0, key, gflag);
    FHG_TRY(scan_exclusive_u32(ws, gflag, gpos, m0, cnt));
    FHG_CUDA(cudaMemcpyAsync(&h, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    const int64_t mu = m0 > 0 ? h : 0;
    const size_t gz = (size_t)(mu > 0 ? mu : 1);
    unsigned long long* gmin;
    int32_t *gu, *gv;
    FHG_TRY(ws.alloc(&gmin, gz));
    FHG_TRY(ws.alloc(&gu, gz));
    FHG_TRY(ws.alloc(&gv, gz));
    LAUNCH(pc_fill_u64_kernel, mu, reinterpret_cast<uint64_t*>(gmin), mu, ~0ull);
    LAUNCH(pc_group_min_kernel, m0, m0, n, key, at, d0, gflag, gpos, gmin, gu, gv);

    // ---- _core_distances_csr
    if (2 * mu > 0x7fffffffLL) {
        set_error("precomputed: %lld symmetric entries exceed the int32 entry index",
                  (long long)(2 * mu));
        return FHG_ERR_UNSUPPORTED;
    }
    int32_t* perm;
    FHG_TRY(ws.alloc(&perm, gz));
    if (mu > 0) {
        Workspace tmp(ws);
        uint32_t *vrow, *ubeg, *lbeg;
        FHG_TRY(tmp.alloc(&vrow, gz));
        FHG_TRY(tmp.alloc(&ubeg, (size_t)(n + 1)));
        FHG_TRY(tmp.alloc(&lbeg, (size_t)(n + 1)));
        LAUNCH(pc_mirror_kernel, mu, mu, gv, vrow, perm);
        if (mu > 1) {
            Workspace sort(tmp);
            FHG_TRY(radix_sort_u32(sort, vrow, perm, mu, 0, bits_for(n)));
        }
        FHG_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t), s));
        LAUNCH(pc_rows_kernel, n + 1, n, mu, gu, vrow, ubeg, lbeg, cnt);
        FHG_CUDA(cudaMemcpyAsync(&h, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        FHG_CUDA(cudaStreamSynchronize(s));
        if (h <= (uint32_t)kPcRow) {
            ::fhg::note_launch();
            pc_rank_rows_kernel<<<grid_for(n, kPcWarps), kPcWarps * 32, 0, s>>>(
                n, k, min_samples, gu, gv, gmin, perm, ubeg, lbeg, neighbors, core);
            FHG_CUDA(cudaGetLastError());
        } else {
            FHG_TRY(core_by_sorting(tmp, n, mu, k, min_samples, gu, gv, gmin, neighbors, core));
        }
    }

    // ---- mutual-reachability weights, stably sorted, and the forest
    uint64_t* mkey;
    int2* uv;
    FHG_TRY(ws.alloc(&mkey, gz));
    FHG_TRY(ws.alloc(&uv, gz));
    LAUNCH(pc_mrd_kernel, mu, mu, gu, gv, gmin, core, mkey, perm);
    if (mu > 1) {
        Workspace tmp(ws);
        FHG_TRY(radix_sort_u64(tmp, mkey, perm, mu, 0, 64));
    }
    LAUNCH(pc_ranks_kernel, mu, mu, perm, gu, gv, uv);
    if (n < 2) return FHG_OK;
    return sorted_forest_edges(ws, n, mu, 0, nullptr, nullptr, uv, nullptr, 0, edges,
                               n_components, reinterpret_cast<const double*>(mkey));
}

}  // namespace fhg
