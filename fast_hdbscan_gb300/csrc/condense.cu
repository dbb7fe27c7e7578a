// Condensed tree (cluster_trees.py:205 condense_tree), in parallel.
//
// The reference walks the linkage tree breadth-first from the root and, at
// every node it reaches, applies one of six cases to the two children
// (cluster_trees.py:263-350) by comparing their sizes with
// min_cluster_size: a child either continues the parent's cluster, starts a
// new cluster (both children large), or is eliminated -- all its points are
// emitted as rows at the parent's lambda (eliminate_branch, :148).
//
// The same decisions are local to each node here; what remains are prefix
// properties along root paths, computed for all nodes at once by pointer
// doubling over the linkage tree:
//   depth and DFS preorder      -> breadth-first order = sort by (depth, preorder)
//   topmost non-continuing node -> whether a node is reached, and for a point
//                                  the node that emits it
//   nearest cluster birth       -> the condensed label of a reached node
// Rows come in the reference's emission order: (emitting node's row offset,
// depth, preorder).  A node's place in the preorder is a number below 2n - 1,
// so the nodes are listed in preorder by writing each at its place, and the
// points of one segment are neighbours in that list.  New cluster
// labels are numbered by a prefix count of "both children large" nodes in
// breadth-first order.
#include "compact.cuh"
#include "primitives.cuh"
#include "trees.cuh"

namespace fhg {
namespace {

enum : int8_t { C1 = 1, C2, C3, C4, C5, C6 };

__device__ __forceinline__ float lambda_of(double d) {
    return (float)(d > 0.0 ? 1.0 / d : (double)INFINITY);
}

// Per internal node: case, lambda, and the child flags written into the
// node-indexed arrays of its two children.  *odd is cleared when a node's size
// is not the sum of its children's.
__global__ void cases_kernel(int64_t m, int64_t n, const int32_t* __restrict__ left,
                             const int32_t* __restrict__ right, const double* __restrict__ w,
                             const int32_t* __restrict__ size, const float* __restrict__ wsize,
                             double mcs, double max_cs, int8_t* __restrict__ kase,
                             float* __restrict__ lam,
                             int32_t* __restrict__ par, int8_t* __restrict__ cont,
                             int8_t* __restrict__ birth, int8_t* __restrict__ side,
                             int32_t* __restrict__ odd) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int32_t L = left[i], R = right[i];
    if ((int64_t)size[n + i] != (int64_t)size[L] + size[R]) *odd = 0;
    // counts: leaves, or the points' sample weights (cluster_trees.py:253-262)
    const double lc = wsize ? (double)wsize[L] : (double)(float)size[L];
    const double rc = wsize ? (double)wsize[R] : (double)(float)size[R];
    int8_t c;
    if (L < n && rc >= mcs) c = C1;
    else if (lc < mcs && rc >= mcs) c = C2;
    else if (lc >= mcs && rc < mcs) c = C3;
    else if (lc < mcs && rc < mcs) c = C4;
    else if (lc > max_cs && rc > max_cs) c = C5;
    else c = C6;
    kase[i] = c;
    lam[i] = lambda_of(w[i]);
    par[L] = (int32_t)i;
    par[R] = (int32_t)i;
    side[L] = 0;
    side[R] = 1;
    cont[L] = (c == C3 || c == C5 || c == C6) ? 1 : 0;
    cont[R] = (c == C1 || c == C2 || c == C5 || c == C6) ? 1 : 0;
    birth[L] = birth[R] = (c == C6) ? 1 : 0;
}

// Pointer-doubling state of internal node i (node id n + i), one 32-byte
// record so that the gather of an ancestor's state touches a single sector:
//   anc  current ancestor (internal index; the root is its own ancestor)
//   dep  edges from the node up to anc;  pre  preorder offset up to anc
//   top  topmost non-continuing node on the path (-1: none yet)
//   bth  nearest cluster birth on the path (-1: none yet)
struct __align__(32) PjRec {
    int32_t anc, dep, top, bth;
    long long pre, pad;
};
__device__ __forceinline__ PjRec pj_load(const PjRec* __restrict__ R, int64_t i) {
    const int4 a = __ldg(reinterpret_cast<const int4*>(R + i));
    const longlong2 b = __ldg(reinterpret_cast<const longlong2*>(R + i) + 1);
    PjRec r;
    r.anc = a.x; r.dep = a.y; r.top = a.z; r.bth = a.w;
    r.pre = b.x; r.pad = 0;
    return r;
}
__device__ __forceinline__ void pj_store(PjRec* R, int64_t i, const PjRec& r) {
    reinterpret_cast<int4*>(R + i)[0] = make_int4(r.anc, r.dep, r.top, r.bth);
    reinterpret_cast<longlong2*>(R + i)[1] = make_longlong2(r.pre, 0);
}

__global__ void pj_init_kernel(int64_t m, int64_t n, const int32_t* __restrict__ par,
                               const int8_t* __restrict__ cont, const int8_t* __restrict__ birth,
                               const int8_t* __restrict__ side, const int32_t* __restrict__ left,
                               const int32_t* __restrict__ size, PjRec* __restrict__ R) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int64_t v = n + i;
    PjRec r;
    if (i == m - 1) {  // root
        r.anc = (int32_t)i;
        r.dep = 0;
        r.pre = 0;
        r.top = -1;
        r.bth = (int32_t)v;
    } else {
        const int32_t p = par[v];
        r.anc = p;
        r.dep = 1;
        r.pre = side[v] == 0 ? 1 : 2 * (long long)size[left[p]];
        r.top = cont[v] ? -1 : (int32_t)v;
        r.bth = birth[v] ? (int32_t)v : -1;
    }
    pj_store(R, i, r);
}

// One step: four paths joined into one, i.e. two doublings (three gathers and
// one record read and written, against two of each).  A node's state covers
// the path from it up to (not including) its ancestor; the root's own
// contribution is an identity for dep, pre and top and a default for bth, so a
// state is final once its ancestor is the root and it has a birth.  `moving`
// (nullable) is set when some state is not.
__global__ void pj_step_kernel(int64_t m, const PjRec* __restrict__ R, PjRec* __restrict__ R2,
                               int* __restrict__ moving) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int32_t root = (int32_t)(m - 1);
    PjRec x = pj_load(R, i);
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        if (x.anc == root && x.bth != -1) break;
        const PjRec y = pj_load(R, x.anc);
        x.anc = y.anc;
        x.dep += y.dep;
        x.pre += y.pre;
        x.top = y.top != -1 ? y.top : x.top;
        x.bth = x.bth != -1 ? x.bth : y.bth;
    }
    if (moving && (x.anc != root || x.bth == -1)) *moving = 1;
    pj_store(R2, i, x);
}

// node_at: the node at every place of the preorder (sizes given with a linkage
// tree that are not its own leave or overstep places: condense_tree starts over).
__global__ void pj_split_kernel(int64_t m, int64_t n, const PjRec* __restrict__ R,
                                int32_t* __restrict__ dep, int64_t* __restrict__ pre,
                                int32_t* __restrict__ top, int32_t* __restrict__ bth,
                                int32_t* __restrict__ node_at) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const PjRec x = pj_load(R, i);
    dep[i] = x.dep;
    pre[i] = x.pre;
    top[i] = x.top;
    bth[i] = x.bth;
    if (x.pre >= 0 && x.pre < n + m) node_at[x.pre] = (int32_t)(n + i);
}

// Points: derive from the parent node; decide the emitting node and segment.
__global__ void points_kernel(int64_t n, int64_t m, const int32_t* __restrict__ par,
                              const int8_t* __restrict__ cont, const int8_t* __restrict__ side,
                              const int32_t* __restrict__ left, const int32_t* __restrict__ size,
                              const int32_t* __restrict__ dep, const int64_t* __restrict__ pre,
                              const int32_t* __restrict__ top, int32_t* __restrict__ emit_u,
                              int8_t* __restrict__ emit_part, int32_t* __restrict__ pdep,
                              int32_t* __restrict__ node_at) {
    int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n) return;
    const int32_t p = par[x];
    pdep[x] = dep[p] + 1;
    const int64_t at = pre[p] + (side[x] == 0 ? 1 : 2 * (int64_t)size[left[p]]);
    if (at >= 0 && at < n + m) node_at[at] = (int32_t)x;
    int32_t t = top[p];
    if (t == -1) t = cont[x] ? -1 : (int32_t)x;
    if (t == -1) {
        emit_u[x] = -1;
        emit_part[x] = 0;
        return;
    }
    emit_u[x] = par[t];
    emit_part[x] = side[t];
}

// Reached internal nodes (no non-continuing node on the path), in preorder.
struct ReachedNodes {
    int64_t n;
    const int32_t *node_at, *top, *dep;
    int32_t* reached;
    uint32_t* key;  // their depths
    __device__ bool test(int64_t j) const {
        const int32_t v = node_at[j];
        return v >= n && top[v - n] == -1;
    }
    __device__ void emit(int64_t j, uint32_t at) const {
        const int32_t i = (int32_t)(node_at[j] - n);
        reached[at] = i;
        key[at] = (uint32_t)dep[i];
    }
    __device__ void each(int64_t) const {}
};
// A reached node's rows and new clusters in one 64-bit word, so that one scan
// gives both offsets.
constexpr int kRowBits = 33;
__device__ __forceinline__ int64_t row_part(int64_t v) { return v & (((int64_t)1 << kRowBits) - 1); }
__device__ __forceinline__ int64_t new_part(int64_t v) { return v >> kRowBits; }
// Row counts and "new clusters" flags of reached nodes in breadth-first order.
__global__ void reached_counts_kernel(int64_t cnt, const int32_t* __restrict__ items,
                                      const int8_t* __restrict__ kase,
                                      const int32_t* __restrict__ left,
                                      const int32_t* __restrict__ right,
                                      const int32_t* __restrict__ size,
                                      int64_t* __restrict__ count,
                                      int32_t* __restrict__ bfs_pos) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cnt) return;
    int32_t i = items[j];
    int8_t c = kase[i];
    int64_t r = 0;
    if (c == C1) r = 1;
    else if (c == C2) r = size[left[i]];
    else if (c == C3) r = size[right[i]];
    else if (c == C4) r = (int64_t)size[left[i]] + size[right[i]];
    else if (c == C6) r = 2;
    count[j] = r | ((int64_t)(c == C6 ? 1 : 0) << kRowBits);
    bfs_pos[i] = (int32_t)j;
}
// Condensed label of every reached node (from its nearest birth).
__global__ void reached_labels_kernel(int64_t cnt, int64_t n, const int32_t* __restrict__ items,
                                      const int32_t* __restrict__ bth,
                                      const int32_t* __restrict__ par,
                                      const int8_t* __restrict__ side,
                                      const int32_t* __restrict__ bfs_pos,
                                      const int64_t* __restrict__ off,
                                      int32_t* __restrict__ label) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cnt) return;
    int32_t i = items[j];
    int32_t b = bth[i];
    const int64_t root_node = 2 * n - 2;
    int32_t lab;
    if (b == (int32_t)root_node) lab = (int32_t)n;
    else {
        int32_t u = par[b];
        lab = (int32_t)(n + 1 + 2 * new_part(off[bfs_pos[u]]) + side[b]);
    }
    label[i] = lab;
}

// The points that get a row, in preorder, each with the row its segment (the
// points eliminated under one child of one node) starts at and its depth.
struct EmittedPoints {
    int64_t n;
    const int32_t *node_at, *emit_u;
    const int8_t *emit_part, *kase;
    const int32_t *left, *size, *bfs_pos, *pdep;
    const int64_t* off;
    int32_t* items;
    uint32_t *kseg, *kdep;
    int64_t room;
    __device__ bool test(int64_t j) const {
        const int32_t x = node_at[j];
        return x >= 0 && x < n && emit_u[x] >= 0;
    }
    __device__ void emit(int64_t j, uint32_t at) const {
        if (at >= room) return;
        const int32_t x = node_at[j], u = emit_u[x];
        int64_t base = row_part(off[bfs_pos[u]]);
        if (emit_part[x] == 1 && kase[u] == C4) base += size[left[u]];
        items[at] = x;
        kseg[at] = (uint32_t)base;
        kdep[at] = (uint32_t)pdep[x];
    }
    __device__ void each(int64_t) const {}
};
__device__ __forceinline__ void point_row(int64_t r, int64_t rows, int32_t x, const int32_t* emit_u,
                                          const int32_t* label, const float* lam,
                                          int32_t* oparent, int32_t* ochild, float* olam,
                                          float* osize) {
    if (r < 0 || r >= rows) return;
    const int32_t u = emit_u[x];
    oparent[r] = label[u];
    ochild[r] = x;
    olam[r] = lam[u];
    osize[r] = 1.0f;
}
// A segment is a run of the preorder, of fewer than min_cluster_size points:
// every point counts the points of its run that precede it by (depth,
// preorder), which is its row.
__global__ void point_rows_kernel(int64_t items_n, int64_t rows, const int32_t* __restrict__ items,
                                  const uint32_t* __restrict__ kseg,
                                  const uint32_t* __restrict__ kdep,
                                  const int32_t* __restrict__ emit_u,
                                  const int32_t* __restrict__ label,
                                  const float* __restrict__ lam, int32_t* __restrict__ oparent,
                                  int32_t* __restrict__ ochild, float* __restrict__ olam,
                                  float* __restrict__ osize) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= items_n) return;
    const uint32_t seg = kseg[t], dep = kdep[t];
    int64_t r = seg;
    for (int64_t j = t - 1; j >= 0 && kseg[j] == seg; --j) r += kdep[j] <= dep ? 1 : 0;
    for (int64_t j = t + 1; j < items_n && kseg[j] == seg; ++j) r += kdep[j] < dep ? 1 : 0;
    point_row(r, rows, items[t], emit_u, label, lam, oparent, ochild, olam, osize);
}
// The same with the rank from a sort (order: items by segment, depth,
// preorder): its place in its run of the sorted segments.
__global__ void gather_u32_kernel(int64_t cnt, const uint32_t* __restrict__ src,
                                  const int32_t* __restrict__ perm, uint32_t* __restrict__ dst) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < cnt) dst[t] = src[perm[t]];
}
__global__ void run_starts_kernel(int64_t items_n, int64_t rows,
                                  const uint32_t* __restrict__ seg, int32_t* __restrict__ start) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < items_n && seg[t] < rows && (t == 0 || seg[t - 1] != seg[t]))
        start[seg[t]] = (int32_t)t;
}
__global__ void sorted_point_rows_kernel(int64_t items_n, int64_t rows, const int32_t* __restrict__ order,
                                         const uint32_t* __restrict__ seg,
                                         const int32_t* __restrict__ start,
                                         const int32_t* __restrict__ items,
                                         const int32_t* __restrict__ emit_u,
                                         const int32_t* __restrict__ label,
                                         const float* __restrict__ lam,
                                         int32_t* __restrict__ oparent,
                                         int32_t* __restrict__ ochild, float* __restrict__ olam,
                                         float* __restrict__ osize) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= items_n || seg[t] >= rows) return;
    const int64_t r = (int64_t)seg[t] + (t - start[seg[t]]);
    point_row(r, rows, items[order[t]], emit_u, label, lam, oparent, ochild, olam, osize);
}
// The two rows of every node that starts clusters.
__global__ void cluster_rows_kernel(int64_t cnt, int64_t n, const int32_t* __restrict__ reached,
                                    const int8_t* __restrict__ kase,
                                    const int64_t* __restrict__ off,
                                    const int32_t* __restrict__ label,
                                    const float* __restrict__ lam,
                                    const int32_t* __restrict__ left,
                                    const int32_t* __restrict__ right,
                                    const int32_t* __restrict__ size,
                                    const float* __restrict__ wsize,
                                    int32_t* __restrict__ oparent, int32_t* __restrict__ ochild,
                                    float* __restrict__ olam, float* __restrict__ osize) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cnt) return;
    const int32_t u = reached[j];
    if (kase[u] != C6) return;
    for (int s = 0; s < 2; ++s) {
        const int64_t r = row_part(off[j]) + s;
        const int32_t v = s == 0 ? left[u] : right[u];
        oparent[r] = label[u];
        ochild[r] = (int32_t)(n + 1 + 2 * new_part(off[j]) + s);
        olam[r] = lam[u];
        osize[r] = wsize ? wsize[v] : (float)size[v];
    }
}

__global__ void condensed_out_kernel(int64_t rows, const int32_t* __restrict__ p,
                                     const int32_t* __restrict__ c, const float* __restrict__ l,
                                     const float* __restrict__ z, int64_t* __restrict__ op,
                                     int64_t* __restrict__ oc, float* __restrict__ ol,
                                     float* __restrict__ oz) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    op[r] = p[r];
    oc[r] = c[r];
    ol[r] = l[r];
    oz[r] = z[r];
}

// Segments of at most this many points are ordered by counting: a point reads
// its whole segment, so longer ones (and those of weighted trees, whose sizes
// are no counts) are sorted.
constexpr int64_t kCountedRun = 512;

#define LAUNCH(kernel, count, ...)                                          \
    do {                                                                    \
        if ((count) > 0) {                                                  \
            ::fhg::note_launch(); \
            kernel<<<grid_for((count), 256), 256, 0, s>>>(__VA_ARGS__);     \
            FHG_CUDA(cudaGetLastError());                                   \
        }                                                                   \
    } while (0)

// Sizes as the weights that the cases go by.
__global__ void sizes_as_weights_kernel(int64_t nodes, const int32_t* __restrict__ size,
                                        float* __restrict__ wsize) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < nodes) wsize[v] = (float)size[v];
}

template <class T>
int read1(const T* dev, T* host, cudaStream_t s) {
    FHG_CUDA(cudaMemcpyAsync(host, dev, sizeof(T), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    return FHG_OK;
}

}  // namespace

int condense_tree(Workspace& ws, const Linkage& lk, int64_t mcs, double max_cs, Condensed* out) {
    cudaStream_t s = ws.stream();
    const int64_t n = lk.n, m = lk.m;
    *out = Condensed();
    out->n = n;
    if (m <= 0) return FHG_OK;
    Stage stage(s, "condense");
    const int64_t nodes = n + m;

    int8_t *kase, *cont, *birth, *side, *emit_part;
    float* lam;
    int32_t *par, *dep, *top, *bth, *emit_u, *pdep, *node_at;
    int64_t* pre;
    FHG_TRY(ws.alloc(&kase, (size_t)m));
    FHG_TRY(ws.alloc(&lam, (size_t)m));
    FHG_TRY(ws.alloc(&par, (size_t)nodes));
    FHG_TRY(ws.alloc(&cont, (size_t)nodes));
    FHG_TRY(ws.alloc(&birth, (size_t)nodes));
    FHG_TRY(ws.alloc(&side, (size_t)nodes));
    // the nodes in preorder, a flag (-1: every size is its children's sum) and the
    // number of reached nodes
    FHG_TRY(ws.alloc(&node_at, (size_t)(nodes + 2)));
    int32_t* odd = node_at + nodes;
    FHG_CUDA(cudaMemsetAsync(node_at, 0xff, sizeof(int32_t) * (nodes + 1), s));
    LAUNCH(cases_kernel, m, m, n, lk.left, lk.right, lk.w, lk.size, lk.wsize, (double)mcs, max_cs,
           kase, lam,
           par, cont, birth, side, odd);

    FHG_TRY(ws.alloc(&dep, (size_t)m));
    FHG_TRY(ws.alloc(&pre, (size_t)m));
    FHG_TRY(ws.alloc(&top, (size_t)m));
    FHG_TRY(ws.alloc(&bth, (size_t)m));
    {
        Workspace tmp(ws);
        PjRec *R, *R2;
        int* moving;
        FHG_TRY(tmp.alloc(&R, (size_t)m));
        FHG_TRY(tmp.alloc(&R2, (size_t)m));
        FHG_TRY(tmp.alloc(&moving, 1));
        LAUNCH(pj_init_kernel, m, m, n, par, cont, birth, side, lk.left, lk.size, R);
        // log4(height) + 1 steps finish every node; the height is not known,
        // so from step 6 on every second step reports whether it was the last
        const int steps = (bits_for(m) + 1) / 2 + 1;
        for (int r = 0; r < steps; ++r) {
            const bool check = r >= 5 && (r & 1) == 1 && r + 1 < steps;
            if (check) FHG_CUDA(cudaMemsetAsync(moving, 0, sizeof(int), s));
            LAUNCH(pj_step_kernel, m, m, R, R2, check ? moving : nullptr);
            std::swap(R, R2);
            if (check) {
                int h_moving = 1;
                FHG_TRY(read1(moving, &h_moving, s));
                if (!h_moving) break;
            }
        }
        LAUNCH(pj_split_kernel, m, m, n, R, dep, pre, top, bth, node_at);
    }

    FHG_TRY(ws.alloc(&emit_u, (size_t)n));
    FHG_TRY(ws.alloc(&emit_part, (size_t)n));
    FHG_TRY(ws.alloc(&pdep, (size_t)n));
    LAUNCH(points_kernel, n, n, m, par, cont, side, lk.left, lk.size, dep, pre, top, emit_u,
           emit_part, pdep, node_at);

    // ---- reached internal nodes in breadth-first order: by depth, stably from
    // the preorder
    uint32_t* kd;
    int32_t *reached, *bfs_pos, *label;
    FHG_TRY(ws.alloc(&reached, (size_t)m));
    FHG_TRY(ws.alloc(&kd, (size_t)m));
    FHG_TRY(compact(ws, ReachedNodes{n, node_at, top, dep, reached, kd}, nodes,
                    reinterpret_cast<uint32_t*>(odd + 1)));
    int2 h_cnt = make_int2(0, 0);
    FHG_CUDA(cudaMemcpyAsync(&h_cnt, odd, sizeof(h_cnt), cudaMemcpyDeviceToHost, s));
    FHG_CUDA(cudaStreamSynchronize(s));
    if (h_cnt.x != -1) {
        // Sizes of the caller's (weight sums without their weights, say): the
        // cases and the rows' sizes go by them, as the reference's do, but places
        // and numbers of rows by the leaves that there are.
        if (lk.wsize) {
            set_error("condense: the linkage is not a tree over its points");
            return FHG_ERR_INVALID;
        }
        Linkage own = lk;
        FHG_TRY(ws.alloc(&own.wsize, (size_t)nodes));
        LAUNCH(sizes_as_weights_kernel, nodes, nodes, lk.size, own.wsize);
        FHG_TRY(linkage_leaf_counts(ws, own));
        return condense_tree(ws, own, mcs, max_cs, out);
    }
    const int64_t cnt = h_cnt.y;
    // (every node above a reached one is reached: no depth is cnt or more)
    FHG_TRY(radix_sort_u32(ws, kd, reached, cnt, 0, bits_for(cnt)));
    int64_t *count, *off, *tot;
    FHG_TRY(ws.alloc(&count, (size_t)cnt));
    FHG_TRY(ws.alloc(&off, (size_t)cnt));
    FHG_TRY(ws.alloc(&tot, 1));
    FHG_TRY(ws.alloc(&bfs_pos, (size_t)m));
    FHG_TRY(ws.alloc(&label, (size_t)m));
    LAUNCH(reached_counts_kernel, cnt, cnt, reached, kase, lk.left, lk.right, lk.size, count,
           bfs_pos);
    FHG_TRY(scan_exclusive_i64(ws, count, off, cnt, tot));
    LAUNCH(reached_labels_kernel, cnt, cnt, n, reached, bth, par, side, bfs_pos, off, label);
    int64_t h_tot = 0;
    FHG_TRY(read1(tot, &h_tot, s));
    const int64_t rows = h_tot & (((int64_t)1 << kRowBits) - 1), births = h_tot >> kRowBits;
    out->rows = rows;
    out->n_clusters = 1 + 2 * births;
    FHG_TRY(ws.alloc(&out->parent, (size_t)(rows > 0 ? rows : 1)));
    FHG_TRY(ws.alloc(&out->child, (size_t)(rows > 0 ? rows : 1)));
    FHG_TRY(ws.alloc(&out->lambda, (size_t)(rows > 0 ? rows : 1)));
    FHG_TRY(ws.alloc(&out->csize, (size_t)(rows > 0 ? rows : 1)));
    if (rows == 0) return FHG_OK;

    // ---- rows: the clusters' own, and the points by (segment, depth, preorder)
    LAUNCH(cluster_rows_kernel, cnt, cnt, n, reached, kase, off, label, lam, lk.left, lk.right,
           lk.size, lk.wsize, out->parent, out->child, out->lambda, out->csize);
    const int64_t pts = rows - 2 * births;
    if (pts <= 0) return FHG_OK;
    Workspace tmp(ws);
    int32_t* items;
    uint32_t *kseg, *kdep;
    FHG_TRY(tmp.alloc(&items, (size_t)pts));
    FHG_TRY(tmp.alloc(&kseg, (size_t)pts));
    FHG_TRY(tmp.alloc(&kdep, (size_t)pts));
    FHG_TRY(compact(tmp, EmittedPoints{n, node_at, emit_u, emit_part, kase, lk.left, lk.size,
                                       bfs_pos, pdep, off, items, kseg, kdep, pts},
                    nodes, nullptr));
    if (!lk.wsize && mcs <= kCountedRun) {
        LAUNCH(point_rows_kernel, pts, pts, rows, items, kseg, kdep, emit_u, label, lam, out->parent,
               out->child, out->lambda, out->csize);
        return FHG_OK;
    }
    int32_t *order, *start;
    uint32_t* key;
    FHG_TRY(tmp.alloc(&order, (size_t)pts));
    FHG_TRY(tmp.alloc(&start, (size_t)rows));
    FHG_TRY(tmp.alloc(&key, (size_t)pts));
    FHG_TRY(fill_iota_i32(order, pts, s));
    FHG_TRY(radix_sort_u32(tmp, kdep, order, pts, 0, bits_for(n)));
    LAUNCH(gather_u32_kernel, pts, pts, kseg, order, key);
    FHG_TRY(radix_sort_u32(tmp, key, order, pts, 0, bits_for(rows)));
    LAUNCH(run_starts_kernel, pts, pts, rows, key, start);
    LAUNCH(sorted_point_rows_kernel, pts, pts, rows, order, key, start, items, emit_u, label, lam,
           out->parent, out->child, out->lambda, out->csize);
    return FHG_OK;
}

int condensed_to_arrays(const Condensed& ct, int64_t* parent, int64_t* child, float* lambda,
                        float* csize, cudaStream_t s) {
    LAUNCH(condensed_out_kernel, ct.rows, ct.rows, ct.parent, ct.child, ct.lambda, ct.csize,
           parent, child, lambda, csize);
    return FHG_OK;
}

}  // namespace fhg
