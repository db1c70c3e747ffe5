// Error type of the host code, device buffers and the pools that they come from.
// Part of lds_host.cu; a header of its own so that the CPU tests can compile it
// against a fake CUDA runtime whose calls fail where a test asks for it.
#pragma once
#include <cstdarg>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>

#include <cuda_runtime_api.h>

#include "../../include/lds.h"

namespace lds {
namespace {

struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

[[noreturn]] void fail(int code, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    throw Error(code, buf);
}

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) fail(LDS_ERR_CUDA, "CUDA error in %s: %s", what, cudaGetErrorString(e));
}

// ---------------------------------------------------------------------------
// Device buffers
// ---------------------------------------------------------------------------
// Owning device allocation; move-only so containers never double-free.
// Stream-ordered allocation target of this thread: while a PoolScope is alive,
// DevBuf allocations come from the library's private memory pool on its stream
// and go back to it with cudaFreeAsync, which (unlike cudaFree) does not wait
// for the whole device; the pool keeps its reservation for later calls.
struct PoolTarget {
    cudaMemPool_t pool = nullptr;
    cudaStream_t st = nullptr;
};
thread_local PoolTarget t_pool;

struct PoolScope {
    PoolTarget saved;
    PoolScope(cudaMemPool_t pool, cudaStream_t st) : saved(t_pool) { t_pool = {pool, st}; }
    ~PoolScope() { t_pool = saved; }
};

// The pool of buffers that live for one call (CallScope), null until first used,
// and the bytes that it has handed out (both change under the context's lock).
// Buffers above kCallPoolBuf, and any that would take it above kCallPoolKeep, are
// ordinary memory: the pool maps new memory at 6 to 70 ms per GB and unmaps what it
// may not keep at as much, where cudaMalloc takes under 1 ms (a GxE right pair of
// 2.6 GB: 728 ms).
cudaMemPool_t g_call_pool = nullptr;
size_t g_call_pool_live = 0;
constexpr size_t kCallPoolBuf = 128ull << 20;
constexpr size_t kCallPoolKeep = 512ull << 20;

struct DevBuf {
    void* p = nullptr;
    size_t n = 0;
    cudaStream_t pool_st = nullptr;  // non-null: pool memory, freed in this stream's order
    bool call_mem = false;           // and of the call pool
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n), pool_st(o.pool_st), call_mem(o.call_mem) {
        o.p = nullptr;
        o.n = 0;
        o.pool_st = nullptr;
        o.call_mem = false;
    }
    DevBuf& operator=(DevBuf&& o) noexcept {
        if (this != &o) {
            release();
            p = o.p;
            n = o.n;
            pool_st = o.pool_st;
            call_mem = o.call_mem;
            o.p = nullptr;
            o.n = 0;
            o.pool_st = nullptr;
            o.call_mem = false;
        }
        return *this;
    }
    // An allocation, from whichever source, that ran out of memory: once more after
    // the call pool has given back what it holds unused.
    template <typename F>
    cudaError_t after_trim(F&& alloc) {
        cudaError_t e = alloc();
        if (e == cudaErrorMemoryAllocation && g_call_pool) {
            cudaGetLastError();
            cudaDeviceSynchronize();
            cudaMemPoolTrimTo(g_call_pool, 0);
            e = alloc();
        }
        if (e != cudaSuccess) p = nullptr;
        return e;
    }
    void* get(size_t bytes) {
        if (bytes <= n && p) return p;
        release();
        if (bytes == 0) bytes = 16;
        const bool call = t_pool.pool && t_pool.pool == g_call_pool;
        if (t_pool.pool && !(call && (bytes > kCallPoolBuf ||
                                      g_call_pool_live + bytes > kCallPoolKeep))) {
            ck(after_trim([&] { return cudaMallocFromPoolAsync(&p, bytes, t_pool.pool, t_pool.st); }),
               "pool allocation");
            pool_st = t_pool.st;
            call_mem = call;
            if (call) g_call_pool_live += bytes;
        } else {
            ck(after_trim([&] { return cudaMalloc(&p, bytes); }), "cudaMalloc");
        }
        n = bytes;
        return p;
    }
    template <typename T>
    T* as(size_t count) { return static_cast<T*>(get(count * sizeof(T))); }
    void release() {
        if (p) {
            if (call_mem) g_call_pool_live -= n;
            if (pool_st) cudaFreeAsync(p, pool_st);
            else cudaFree(p);
        }
        p = nullptr;
        n = 0;
        pool_st = nullptr;
        call_mem = false;
    }
    ~DevBuf() { release(); }
};

// A buffer kept from call to call: ordinary device memory in every scope.
struct KeptBuf : DevBuf {
    void* get(size_t bytes) {
        PoolScope plain(nullptr, nullptr);
        return DevBuf::get(bytes);
    }
    template <typename T>
    T* as(size_t count) { return static_cast<T*>(get(count * sizeof(T))); }
};

}  // namespace
}  // namespace lds
