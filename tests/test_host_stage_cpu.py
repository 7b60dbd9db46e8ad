"""Device-to-host copies of a handle on another GPU than the caller's (rs_host_stage.h), built
against a runtime of two fake GPUs: the caller's device is the same after every call, streams,
events and synchronisations belong to the handle's device, and the bytes arrive, whether the
copy takes the threads' path, the plain one, or fails."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rayspace3d_gb300", "csrc")

RUNTIME = r"""
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <cstring>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyDeviceToHost = 2 };
enum { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum { cudaStreamNonBlocking = 1, cudaEventDisableTiming = 2 };
struct cudaPointerAttributes { int type = 0; };
struct Owned { int device; };
using cudaStream_t = Owned*;
using cudaEvent_t = Owned*;
inline thread_local int current = 0;           // the thread's device
inline std::atomic<int> wrong{0};              // work on another device than its object's
inline std::atomic<int> copies{0}, fail_copy{-1}, live{0};
inline int handle_device = 1;
inline bool fail_pinned = false;
inline int dst_type = cudaMemoryTypeUnregistered;
inline cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = dst_type; return cudaSuccess; }
inline cudaError_t make(Owned** o) { *o = new Owned{current}; ++live; if (current != handle_device) ++wrong; return cudaSuccess; }
inline cudaError_t drop(Owned* o) { delete o; --live; return cudaSuccess; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, int) { return make(s); }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { return make(e); }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s); }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e); }
inline cudaError_t cudaMallocHost(void** p, size_t n) {
    if (fail_pinned) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    ++live;
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) { std::free(p); --live; return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (current != (s ? s->device : handle_device)) ++wrong; return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { if (e->device != s->device) ++wrong; return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (current != st->device || st->device != handle_device) ++wrong;
    if (copies++ == fail_copy) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
"""

MAIN = r"""
#include "rs_host_stage.h"
#include <cstdio>
#include <vector>
static int check(const char* what, size_t bytes, int caller, int handle, bool ok) {
    current = caller;
    handle_device = handle;
    copies = 0;
    std::vector<unsigned char> src(bytes), dst(bytes, 0);
    for (size_t i = 0; i < bytes; ++i) src[i] = (unsigned char)(i * 2654435761u >> 24);
    int bad = 0;
    {
        rs::HostStage stage;
        for (int rep = 0; rep < 2; ++rep) {
            const cudaError_t e = stage.copy(dst.data(), src.data(), bytes, handle);
            if ((e == cudaSuccess) != ok) bad |= 1;
            if (ok && dst != src) bad |= 2;
            if (current != caller) bad |= 4;
            if (wrong != 0) bad |= 8;
            wrong = 0;
            std::fill(dst.begin(), dst.end(), 0);
            copies = 0;
        }
    }
    if (live != 0) bad |= 16;
    std::printf("%s %d\n", what, bad);
    return bad;
}
int main() {
    const size_t big = (size_t(23) << 20) + 12345;
    int bad = 0;
    for (int caller = 0; caller < 2; ++caller)
        for (int handle = 0; handle < 2; ++handle) {
            bad |= check("threads", big, caller, handle, true);
            bad |= check("plain", 4096, caller, handle, true);
            dst_type = cudaMemoryTypeHost;
            bad |= check("pinned", big, caller, handle, true);
            dst_type = cudaMemoryTypeUnregistered;
            fail_pinned = true;
            bad |= check("no pinned memory", big, caller, handle, true);
            fail_pinned = false;
            for (int at : {0, 7, 20}) {
                fail_copy = at;
                bad |= check("failed copy", big, caller, handle, false);
                fail_copy = -1;
            }
        }
    return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_callers_device_is_kept(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
