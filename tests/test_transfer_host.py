"""Copies from and to pageable memory (transfer.cu) on the CPU, with fakes of
the CUDA calls: the bytes arrive whatever pinned memory can be had, and the
contexts of a device share a bounded number of chunks, which the last of them
gives back."""

import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

PROGRAM = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstring>
#include <vector>
#include <atomic>
#include <thread>
static std::atomic<int> pins_left, pinned, plain;
static cudaError_t fake_pin(void** p, size_t n, unsigned) {
    if (pins_left <= 0) return cudaErrorMemoryAllocation;
    --pins_left; ++pinned; *p = ::operator new(n);
    return cudaSuccess;
}
static cudaError_t fake_unpin(void* p) { ::operator delete(p); --pinned; return cudaSuccess; }
static cudaError_t fake_copy(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (n > (size_t(1) << 20)) ++plain;
    memcpy(d, s, n);
    return cudaSuccess;
}
static cudaError_t fake_attributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
static cudaError_t ok() { return cudaSuccess; }
#define cudaHostAlloc(p, n, f) fake_pin(p, n, f)
#define cudaFreeHost(p) fake_unpin(p)
#define cudaMemcpyAsync(d, s, n, k, st) fake_copy(d, s, n, k, st)
#define cudaPointerGetAttributes(a, p) fake_attributes(a, p)
#define cudaEventCreateWithFlags(e, f) ok()
#define cudaEventDestroy(e) ok()
#define cudaEventRecord(e, s) ok()
#define cudaEventSynchronize(e) ok()
#define cudaStreamSynchronize(s) ok()
#define cudaSetDevice(d) ok()
#define cudaGetLastError() ok()
#include "transfer.cu"

static bool both_ways(size_t n) {
    prt_ctx ctx;
    prt::transfer_open(0);
    std::vector<char> a(n), b(n), c(n);
    for (size_t i = 0; i < n; ++i) a[i] = (char)(i * 2654435761u >> 13);
    const bool good = prt::copy_in(&ctx, b.data(), a.data(), n) == cudaSuccess &&
                      prt::copy_out(&ctx, c.data(), b.data(), n) == cudaSuccess && c == a;
    prt::transfer_close(0);
    return good;
}

// Copies of `threads` contexts at a time: the most chunks that were pinned.
static int together(int threads) {
    pins_left = 1000;
    std::atomic<int> bad{0};
    std::vector<std::thread> th;
    prt::transfer_open(0);
    for (int i = 0; i < threads; ++i)
        th.emplace_back([&] {
            for (int r = 0; r < 5; ++r) bad += !both_ways((size_t(6) << 20) + 11 * r);
        });
    for (auto& t : th) t.join();
    const int most = pinned;  // chunks stay while a context is open
    prt::transfer_close(0);
    return bad || pinned ? -1 : most;
}

int main() {
    const size_t big = (size_t(9) << 20) + 77;
    for (int left : {100, 1, 0}) {  // every chunk, one chunk and none can be pinned
        pins_left = left;
        plain = 0;
        if (!both_ways(big) || pinned != 0 || plain != (left ? 0 : 2)) { printf("pins %d\n", left); return 1; }
    }
    pins_left = 100;
    plain = 0;
    if (!both_ways((size_t(4) << 20) - 1) || plain != 2 || pins_left != 100) return 2;  // a small copy
    for (int threads : {1, 12}) {
        const int most = together(threads);
        if (most < 1 || most > (threads == 1 ? 8 : 32)) { printf("%d: %d\n", threads, most); return 3; }
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_copies_arrive_with_and_without_pinned_chunks(tmp_path):
    src = tmp_path / "copies.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "copies"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1",
                    "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-o", str(exe), str(src), "-lpthread"], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
