// Shared helpers for the GB300 HDBSCAN engine (sm_103a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/fhg.h"

namespace fhg {

// Last error message of the calling host thread (read by fhg_last_error()).
void set_error(const char* fmt, ...);
const char* last_error();

// Counts every kernel launch made by the library (read by fhg_launch_count).
void note_launch();

// Per-stage timer: when profiling is on (fhg_profile_enable), records a pair
// of CUDA events on the stage's stream; fhg_profile_report sums them by name.
class Stage {
  public:
    Stage(cudaStream_t s, const char* name);
    ~Stage();
    Stage(const Stage&) = delete;
    Stage& operator=(const Stage&) = delete;

  private:
    cudaStream_t s_;
    const char* name_;
    cudaEvent_t a_ = nullptr;
};

// With profiling on, adds `value` to the named counter; fhg_profile_report
// lists it beside the stages as [sum, samples].
void profile_count(const char* name, double value);

// A status carried through the host driver code.  Device kernels never trap:
// bounded loops report through a device status word instead.
struct Status {
    int code = FHG_OK;
    bool ok() const { return code == FHG_OK; }
};

#define FHG_CUDA(expr)                                                                  \
    do {                                                                                \
        cudaError_t _e = (expr);                                                        \
        if (_e != cudaSuccess) {                                                        \
            ::fhg::set_error("%s failed at %s:%d: %s", #expr, __FILE__, __LINE__,      \
                             cudaGetErrorString(_e));                                   \
            return (_e == cudaErrorMemoryAllocation) ? FHG_ERR_OOM : FHG_ERR_CUDA;      \
        }                                                                               \
    } while (0)

#define FHG_TRY(expr)                      \
    do {                                   \
        int _s = (expr);                   \
        if (_s != FHG_OK) return _s;       \
    } while (0)

// The library's stream-ordered memory pool on the current device.  Freed
// blocks stay cached in the pool (release threshold: unlimited), so that the
// synchronisations inside a fit never hand memory back to the driver and the
// next allocation never has to map it again; fhg_release_cached_memory()
// returns the cached blocks.
int device_pool(cudaMemPool_t* out);

// Stream-ordered scratch.  Every buffer of a call is released on the same
// stream when the Workspace goes out of scope.
//
// Buffers of up to a quarter of a block are carved from blocks that the
// Workspace takes from the pool (1 MiB, then twice the last, at most 16 MiB);
// larger ones are their own allocation.  A fit has about a hundred buffers,
// and an allocation with its release costs 0.5 us on one thread but 3.5 us
// per call when 16 threads run fits side by side.
//
// A Workspace made from another one is scratch inside it: its small buffers
// come from the same blocks and their room is used again when it ends, up to
// the last buffer that its parent took meanwhile.  Such Workspaces nest.
class Workspace {
  public:
    explicit Workspace(cudaStream_t s) : stream_(s), arena_(&own_) {}
    explicit Workspace(Workspace& parent)
        : stream_(parent.stream_), pool_(parent.pool_), arena_(parent.arena_) {
        mark_block_ = arena_->blocks.size();
        mark_ = arena_->used;
        level_ = ++arena_->depth;
    }
    ~Workspace() { release(); }
    Workspace(const Workspace&) = delete;
    Workspace& operator=(const Workspace&) = delete;

    template <class T>
    int alloc(T** out, size_t count) {
        size_t bytes = (count * sizeof(T) + kAlign - 1) / kAlign * kAlign;
        if (bytes == 0) bytes = kAlign;
        void* p = nullptr;
        if (bytes > kFirstBlock / 4 && bytes > arena_->size / 4) {
            FHG_TRY(take(&p, bytes));
            bufs_.push_back(p);
        } else {
            if (arena_->used + bytes > arena_->size) {
                const size_t want = arena_->size == 0              ? kFirstBlock
                                    : arena_->size < kLargestBlock ? 2 * arena_->size
                                                                   : kLargestBlock;
                FHG_TRY(take(&p, want));
                arena_->blocks.push_back(p);
                arena_->size = want;
                arena_->used = 0;
            }
            p = static_cast<char*>(arena_->blocks.back()) + arena_->used;
            arena_->used += bytes;
            if (level_ < arena_->depth) {  // outlives the Workspaces inside this one
                arena_->kept_block = arena_->blocks.size();
                arena_->kept = arena_->used;
            }
        }
        *out = static_cast<T*>(p);
        return FHG_OK;
    }
    void release() {
        for (size_t i = bufs_.size(); i-- > 0;) cudaFreeAsync(bufs_[i], stream_);
        bufs_.clear();
        if (arena_ != &own_) {
            if (level_ == 0) return;  // released already
            --arena_->depth;
            level_ = 0;
            if (arena_->blocks.size() == mark_block_) {
                const bool kept = arena_->kept_block == mark_block_ && arena_->kept > mark_;
                arena_->used = kept ? arena_->kept : mark_;
            }
            return;
        }
        for (size_t i = own_.blocks.size(); i-- > 0;) cudaFreeAsync(own_.blocks[i], stream_);
        own_ = Arena();
    }
    cudaStream_t stream() const { return stream_; }

  private:
    static constexpr size_t kAlign = 256, kFirstBlock = size_t{1} << 20,
                            kLargestBlock = size_t{1} << 24;
    struct Arena {
        std::vector<void*> blocks;      // the last one is being filled
        size_t size = 0, used = 0;      // of the last block
        int depth = 0;                  // Workspaces inside
        size_t kept_block = 0, kept = 0;  // room up to here stays taken
    };
    int take(void** p, size_t bytes) {
        if (!pool_) FHG_TRY(device_pool(&pool_));
        cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool_, stream_);
        if (e != cudaSuccess) {
            set_error("cudaMallocFromPoolAsync(%zu bytes) failed: %s", bytes,
                      cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? FHG_ERR_OOM : FHG_ERR_CUDA;
        }
        return FHG_OK;
    }

    cudaStream_t stream_;
    cudaMemPool_t pool_ = nullptr;
    Arena own_;
    Arena* arena_;
    int level_ = 0;
    size_t mark_block_ = 0, mark_ = 0;
    std::vector<void*> bufs_;
};

inline unsigned grid_for(int64_t n, int block) {
    int64_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > 0x7fffffff) g = 0x7fffffff;
    return (unsigned)g;
}

// Monotone float <-> uint32 for non-negative floats (including +inf).
__host__ __device__ inline uint32_t fbits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
__host__ __device__ inline float bitsf(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}

constexpr int kLeaf = 32;     // points per spatial bucket (one warp)
constexpr unsigned kFull = 0xffffffffu;

}  // namespace fhg
