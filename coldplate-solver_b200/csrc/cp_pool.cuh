// Device and pinned host memory of the solver objects.
//
// An object (a flow context, a thermal context, a batch) holds 10 to 200 arrays.
// Allocating and freeing each of them costs more than many solves: a context at
// 811 x 389 took 41 ms to make and destroy for a solve of 110 ms, and now and
// then seconds.  So an object's arrays are cut from blocks, and a destroyed
// object's blocks go to a process-wide cache that the next object takes from.
//   * The cache is bounded (kPoolDeviceMax, kPoolHostMax a CUDA context, or
//     what cp_set_cached_memory_limit() says, 0 for no cache): the oldest
//     blocks beyond that are freed.  It is given back when an allocation of
//     this library fails, before that is tried again, and by
//     cp_release_cached_memory(): other allocators of the process cannot ask
//     for it.
//   * A block is handed on only after its last owner's stream was synchronised
//     (the destroy functions do), so no stream can still be using it, and every
//     array is cleared on its new owner's stream like a fresh one.
//   * A block belongs to the CUDA context it was allocated in, told by the
//     context's id: after cudaDeviceReset, say, the old blocks are not handed
//     out any more (they went with their context), and a block of another
//     device's context waits until that one is current.
//   * One mutex; any thread may create and destroy objects.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <new>
#include <vector>

namespace cp {

constexpr size_t kPoolDeviceMax = size_t(4) << 30;
constexpr size_t kPoolHostMax = size_t(256) << 20;

struct PoolBlock {
    void* p = nullptr;
    size_t bytes = 0;
    unsigned long long ctx = 0;   // id of the CUDA context the block lives in
};

// id of the current CUDA context, unique over the process's life; false if
// there is none
inline bool pool_context(unsigned long long* id) {
    typedef CUresult (*CurrentFn)(CUcontext*);
    typedef CUresult (*IdFn)(CUcontext, unsigned long long*);
    static CurrentFn current = nullptr;
    static IdFn ctxId = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            current = reinterpret_cast<CurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            ctxId = reinterpret_cast<IdFn>(f);
    });
    CUcontext c = nullptr;
    if (!current || !ctxId || cudaFree(nullptr) != cudaSuccess) return false;   // cudaFree(0) makes the context
    return current(&c) == CUDA_SUCCESS && c && ctxId(c, id) == CUDA_SUCCESS;
}

class BlockCache {
public:
    BlockCache(bool host, size_t most) : host_(host), most_(most) {}

    cudaError_t acquire(size_t bytes, PoolBlock* out) {
        unsigned long long ctx = 0;
        const bool known = pool_context(&ctx);
        if (known) {
            std::lock_guard<std::mutex> lock(mutex_);
            size_t best = free_.size();
            for (size_t q = 0; q < free_.size(); ++q) {
                const PoolBlock& b = free_[q];
                if (b.ctx != ctx || b.bytes < bytes || b.bytes > bytes + std::max<size_t>(bytes / 4, size_t(4) << 20)) continue;
                if (best == free_.size() || b.bytes < free_[best].bytes) best = q;
            }
            if (best < free_.size()) {
                *out = free_[best];
                free_.erase(free_.begin() + (long)best);
                return cudaSuccess;
            }
        }
        void* p = nullptr;
        cudaError_t e = alloc(&p, bytes);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            release_all();
            e = alloc(&p, bytes);
        }
        if (e != cudaSuccess) {
            cudaGetLastError();   // reported here; the next launch's check must not find it
            return e;
        }
        *out = PoolBlock{p, bytes, known ? ctx : 0};
        return cudaSuccess;
    }

    // a block that no stream uses any more
    void give(const PoolBlock& b) {
        unsigned long long ctx = 0;
        if (!b.p) return;
        if (!pool_context(&ctx) || b.ctx == 0 || b.ctx != ctx) {
            dealloc(b.p);   // its context is not the current one: an error if it is gone, as before
            cudaGetLastError();
            return;
        }
        bool kept = false;
        try {
            std::lock_guard<std::mutex> lock(mutex_);
            free_.push_back(b);
            kept = true;
        } catch (const std::bad_alloc&) {   // no host memory for the list: the destroy functions do not throw
        }
        if (kept) trim(ctx, false);
        else dealloc(b.p);
    }

    void release_all() {
        unsigned long long ctx = 0;
        if (pool_context(&ctx)) trim(ctx, true);
    }

    // other contexts' blocks are held to it when the next one is given
    void set_limit(size_t bytes) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            most_ = bytes;
        }
        unsigned long long ctx = 0;
        if (pool_context(&ctx)) trim(ctx, false);
    }

private:
    // frees the context's oldest blocks beyond the limit, or all of them
    void trim(unsigned long long ctx, bool all) {
        for (;;) {
            PoolBlock old;
            {
                std::lock_guard<std::mutex> lock(mutex_);
                size_t held = 0, first = free_.size();
                for (size_t q = free_.size(); q-- > 0;)
                    if (free_[q].ctx == ctx) {
                        held += free_[q].bytes;
                        first = q;
                    }
                if (first == free_.size() || (!all && held <= most_)) return;
                old = free_[first];
                free_.erase(free_.begin() + (long)first);
            }
            dealloc(old.p);
        }
    }
    cudaError_t alloc(void** p, size_t bytes) { return host_ ? cudaMallocHost(p, bytes) : cudaMalloc(p, bytes); }
    void dealloc(void* p) {
        if (host_) cudaFreeHost(p);
        else cudaFree(p);
    }
    const bool host_;
    size_t most_;
    std::mutex mutex_;
    std::vector<PoolBlock> free_;   // oldest first
};

// The caches live to the process's end: their blocks go with the CUDA context,
// which is torn down before static destructors could free them safely.
inline BlockCache& device_cache() {
    static BlockCache* c = new BlockCache(false, kPoolDeviceMax);
    return *c;
}
inline BlockCache& host_cache() {
    static BlockCache* c = new BlockCache(true, kPoolHostMax);
    return *c;
}

// The blocks of one object; arrays are cut from them in order, 256-byte
// aligned.  Arrays of 16 MB and more get a block each; smaller ones share
// blocks that grow with the object, from 4 to 32 MB.
class Arena {
public:
    cudaError_t take(size_t bytes, void** out) {
        bytes = (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
        if (bytes > left_) {
            const size_t mb2 = size_t(2) << 20;
            const bool own = bytes >= size_t(16) << 20;
            const size_t want = own ? bytes : std::max(bytes, std::min<size_t>(size_t(32) << 20, std::max<size_t>(size_t(4) << 20, total_)));
            PoolBlock b;
            const cudaError_t e = device_cache().acquire((want + mb2 - 1) / mb2 * mb2, &b);
            if (e != cudaSuccess) return e;
            blocks_.push_back(b);
            total_ += b.bytes;
            if (own) {
                *out = b.p;
                return cudaSuccess;
            }
            cur_ = static_cast<char*>(b.p);
            left_ = b.bytes;
        }
        *out = cur_;
        cur_ += bytes;
        left_ -= bytes;
        return cudaSuccess;
    }
    // the owner's stream must be idle
    void give_back() {
        for (const PoolBlock& b : blocks_) device_cache().give(b);
        blocks_.clear();
        cur_ = nullptr;
        left_ = total_ = 0;
    }

private:
    std::vector<PoolBlock> blocks_;
    char* cur_ = nullptr;
    size_t left_ = 0, total_ = 0;
};

}  // namespace cp
