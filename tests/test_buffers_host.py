"""The host code's device buffers and column transfers, compiled from the library's
own header with the host compiler against a fake CUDA runtime, whose calls fail
where the test asks for it."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

FAKE = r"""
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "lds_buffers.h"

// Device memory of `room` bytes, of which pools hold `kept` unused; the copy that
// counts fail_copy down to zero fails.
static size_t room = 1000, kept = 0;
static int fail_copy = -1, trims = 0;
static cudaError_t take(void** p, size_t n) {
    if (n + kept > room) return cudaErrorMemoryAllocation;
    *p = std::malloc(n ? n : 1);
    return cudaSuccess;
}
static cudaError_t copied() {
    return fail_copy >= 0 && fail_copy-- == 0 ? cudaErrorIllegalAddress : cudaSuccess;
}
extern "C" {
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t CUDARTAPI cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return take(p, n); }
cudaError_t CUDARTAPI cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t CUDARTAPI cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemPoolTrimTo(cudaMemPool_t, size_t) { kept = 0; ++trims; return cudaSuccess; }
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t CUDARTAPI cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemset2DAsync(void* p, size_t ld, int v, size_t w, size_t h, cudaStream_t) {
    for (size_t i = 0; i < h; ++i) std::memset((char*)p + i * ld, v, w);
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpy2DAsync(void* d, size_t dl, const void* s, size_t sl, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t) {
    if (copied() != cudaSuccess) return cudaErrorIllegalAddress;
    for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dl, (const char*)s + i * sl, w);
    return cudaSuccess;
}
}
using namespace lds;
static int bad(const char* what) { std::printf("%s", what); return 0; }
"""


def run_cpp(tmp_path, body: str) -> str:
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(FAKE + body)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wno-unused-function", "-I", str(CUDA), "-I",
                    str(ROOT / "summit_b200" / "csrc"), str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout


needs_cuda_headers = pytest.mark.skipif(not (CUDA / "cuda_runtime_api.h").exists(),
                                        reason="no CUDA headers")


# Memory that the call pool holds unused is given back to whichever allocation runs
# out: ordinary memory, another pool's (the streamed windowed call's) or its own.
@needs_cuda_headers
def test_a_failing_allocation_gets_the_call_pools_memory(tmp_path):
    assert run_cpp(tmp_path, r"""
int main() {
    g_call_pool = (cudaMemPool_t)8;
    cudaMemPool_t pools[] = {nullptr, (cudaMemPool_t)16, g_call_pool};
    for (cudaMemPool_t pool : pools) {
        kept = 600, trims = 0;
        PoolScope scope(pool, (cudaStream_t)4);
        DevBuf b;
        try { b.get(500); } catch (const Error&) { return bad("refused"); }
        if (trims != 1 || !b.p) return bad("not trimmed");
        b.release();
        try { b.get(2000); return bad("too much"); } catch (const Error&) {}
        if (b.p || b.n || g_call_pool_live) return bad("left over");
    }
    g_call_pool = nullptr;
    kept = 600;
    DevBuf b;
    try { b.get(500); return bad("no pool to trim"); } catch (const Error&) {}
    return bad("ok");
}
""") == "ok"


# A block's contribution of several pieces (columns longer than a half; a last partial
# piece) and of one: merged as the sketch's bins ask for, and not at all, nor marked
# as written, where any of its copies fails.
@needs_cuda_headers
@pytest.mark.parametrize("N,K,v,fails", [(300007, 3, 13, [0, 1, 3, 38]), (60001, 3, 50, [0, 5]),
                                         (60001, 3, 7, [0]), (500, 3, 7, [0])])
def test_a_failed_download_leaves_the_sketch(tmp_path, N, K, v, fails):
    assert run_cpp(tmp_path, r"""
int main() {
    const int64_t N = %d, K = %d, v = %d, ld = N + 5;
    std::vector<double> d((size_t)(ld * K * v));
    for (size_t i = 0; i < d.size(); ++i) d[i] = (double)(i %% 1013) - 500.0;
    const std::vector<int64_t> nnz = {3, 5, 0};   // (the last bin has no members)
    PinnedStage stage;
    for (int f : {%s, -1}) {
        std::vector<float> x((size_t)(N * K * v));
        for (size_t i = 0; i < x.size(); ++i) x[i] = (float)(i %% 7);
        const std::vector<float> before = x;
        uint8_t init[3] = {0, 1, 0};
        fail_copy = f;
        bool threw = false;
        try {
            merge_sketch<float>(stage, nullptr, d.data(), ld, N, K, v, nnz.data(), init, x.data());
        } catch (const Error&) { threw = true; }
        if (threw != (f >= 0)) return bad("error not passed on");
        if (threw && (x != before || init[0] != 0 || init[1] != 1)) return bad("changed");
        if (threw) continue;
        for (int64_t q = 0; q < K * v; ++q)
            for (int64_t n = 0; n < N; ++n) {
                const int64_t k = q / v;
                const float old = before[(size_t)(q * N + n)], c = (float)d[(size_t)(q * ld + n)];
                const float want = k == 0 ? c : k == 1 ? old + c : old;
                if (x[(size_t)(q * N + n)] != want) return bad("wrong sum");
            }
        if (init[0] != 1 || init[1] != 1 || init[2] != 0) return bad("marks");
    }
    // and up again: pieces, the padding rows zero
    std::vector<float> h((size_t)(N * K * v));
    for (size_t i = 0; i < h.size(); ++i) h[i] = (float)(i %% 911);
    upload_cols<float>(stage, nullptr, d.data(), ld, h.data(), N, K * v);
    for (int64_t q = 0; q < K * v; ++q)
        for (int64_t n = 0; n < ld; ++n)
            if (d[(size_t)(q * ld + n)] != (n < N ? (double)h[(size_t)(q * N + n)] : 0.0)) return bad("upload");
    return bad("ok");
}
""" % (N, K, v, ", ".join(map(str, fails)))) == "ok"
