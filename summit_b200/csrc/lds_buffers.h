// Error type of the host code, device buffers and the pools that they come from.
// Part of lds_host.cu; a header of its own so that the CPU tests can compile it
// against a fake CUDA runtime whose calls fail where a test asks for it.
#pragma once
#include <algorithm>
#include <cstdarg>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <memory>
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
// 2.6 GB: 728 ms).  Below kCallPoolBuf the pool is the faster one from the first call
// on: GxE reference of 20,000 samples and SNPs, 4 exposures, first and later runs
// 5.2 / 2.75 ms, with only buffers up to 8 MB pooled 6.0 / 4.4; windowed LD of
// 50,000 x 12,000 4.4 / 4.15 and 5.1 / 4.9.
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

// ---------------------------------------------------------------------------
// Columns of doubles between a device array (ld >= rows) and host code that
// converts or merges them, through pinned memory: pieces of whole columns in two
// halves, so that one piece crosses PCIe while the host works on the other.
// ---------------------------------------------------------------------------
constexpr size_t kStageBytes = 2ull << 20;     // a half, or one column where that is longer
constexpr size_t kStageWhole = 64ull << 20;    // a download of up to this many bytes is one piece

struct PinnedStage {
    void* p = nullptr;
    size_t n = 0;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    // At least `bytes`, in halves; no copy of an earlier use is in flight afterwards.
    void reserve(size_t bytes, cudaStream_t st) {
        for (cudaEvent_t& e : ev)
            if (!e) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
        ck(cudaStreamSynchronize(st), "staging");
        if (n >= bytes) return;
        release();
        ck(cudaHostAlloc(&p, bytes, cudaHostAllocDefault), "pinned staging");
        n = bytes;
    }
    double* half(int64_t i) const {
        return reinterpret_cast<double*>(static_cast<char*>(p) + (i & 1 ? n / 2 / 8 * 8 : 0));
    }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        n = 0;
    }
};

// Columns of `rows` doubles in a half.
inline int64_t reserve_halves(PinnedStage& s, int64_t rows, cudaStream_t st) {
    const size_t col = sizeof(double) * (size_t)std::max<int64_t>(rows, 1);
    const size_t half = std::max(kStageBytes, col);
    s.reserve(2 * half, st);
    return std::max<int64_t>(1, (int64_t)(half / col));
}

// The columns on the host, `rows` apart, once all of them have arrived: in the stage,
// which takes up to kStageWhole bytes of them at once, or copied out of its halves to
// `spill` (60,000 x 60, 29 MB, four phase-1 calls and phase 2:
// 53 ms by way of `spill`, 29 in the stage).
inline const double* download_cols(PinnedStage& s, cudaStream_t st, const double* d, int64_t ld,
                                   int64_t rows, int64_t cols, std::unique_ptr<double[]>& spill) {
    const size_t w = sizeof(double) * (size_t)rows;
    auto copy = [&](double* h, int64_t q0, int64_t n) {
        ck(cudaMemcpy2DAsync(h, w, d + q0 * ld, sizeof(double) * (size_t)ld, w, (size_t)n,
                             cudaMemcpyDeviceToHost, st),
           "D2H");
    };
    if (w * (size_t)cols <= kStageWhole) {
        s.reserve(std::max(2 * kStageBytes, w * (size_t)cols), st);
        copy(s.half(0), 0, cols);
        ck(cudaStreamSynchronize(st), "download");
        return s.half(0);
    }
    const int64_t per = reserve_halves(s, rows, st), pieces = (cols + per - 1) / per;
    spill.reset(new double[(size_t)(rows * cols)]);
    auto fetch = [&](int64_t i) {
        copy(s.half(i), i * per, std::min(per, cols - i * per));
        ck(cudaEventRecord(s.ev[i & 1], st), "event");
    };
    for (int64_t i = 0; i < std::min<int64_t>(2, pieces); ++i) fetch(i);
    for (int64_t i = 0; i < pieces; ++i) {
        ck(cudaEventSynchronize(s.ev[i & 1]), "download");
        std::copy_n(s.half(i), (size_t)(std::min(per, cols - i * per) * rows),
                    spill.get() + i * per * rows);
        if (i + 2 < pieces) fetch(i + 2);
    }
    return spill.get();
}

// Columns h (T, `rows` apart) to d as FP64, rows..ld of each column zero.
template <typename T>
void upload_cols(PinnedStage& s, cudaStream_t st, double* d, int64_t ld, const T* h, int64_t rows,
                 int64_t cols) {
    if (cols <= 0) return;
    if (ld > rows)
        ck(cudaMemset2DAsync(d + rows, sizeof(double) * (size_t)ld, 0,
                             sizeof(double) * (size_t)(ld - rows), (size_t)cols, st),
           "memset");
    const int64_t per = reserve_halves(s, rows, st), pieces = (cols + per - 1) / per;
    for (int64_t i = 0; i < pieces; ++i) {
        const int64_t q0 = i * per, n = std::min(per, cols - q0);
        double* p = s.half(i);
        if (i >= 2) ck(cudaEventSynchronize(s.ev[i & 1]), "upload");
        for (int64_t x = 0; x < n * rows; ++x) p[x] = (double)h[q0 * rows + x];
        ck(cudaMemcpy2DAsync(d + q0 * ld, sizeof(double) * (size_t)ld, p,
                             sizeof(double) * (size_t)rows, sizeof(double) * (size_t)rows, (size_t)n,
                             cudaMemcpyHostToDevice, st),
           "H2D");
        ck(cudaEventRecord(s.ev[i & 1], st), "event");
    }
}

// A block's contribution d (K bins x v columns) into the caller's sketch: added to a
// bin that has been written (bin_init null: all have), stored into one that has not;
// bins without members (nnz) are left alone.  Nothing of the caller's changes until
// the whole contribution is on the host, so that a failed call can be repeated.
template <typename T>
void merge_sketch(PinnedStage& s, cudaStream_t st, const double* d, int64_t ld, int64_t N, int64_t K,
                  int64_t v, const int64_t* nnz, uint8_t* bin_init, T* Xz) {
    std::unique_ptr<double[]> spill;
    const double* p = download_cols(s, st, d, ld, N, K * v, spill);
    for (int64_t k = 0; k < K; ++k) {
        if (nnz[k] == 0) continue;
        T* dst = Xz + k * v * N;
        const double* src = p + k * v * N;
        if (!bin_init || bin_init[k])
            for (int64_t x = 0; x < v * N; ++x) dst[x] = (T)((double)dst[x] + src[x]);
        else
            for (int64_t x = 0; x < v * N; ++x) dst[x] = (T)src[x];
        if (bin_init) bin_init[k] = 1;
    }
}

}  // namespace
}  // namespace lds
