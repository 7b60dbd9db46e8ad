// rs_host_stage.h -- copies of large arrays from the device to pageable host memory.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>

#include <cuda_runtime.h>

namespace rs {
// Device to pageable host copies of large arrays: threads that each copy every kThreads-th
// chunk into pinned memory, two chunks in flight, and from there to the caller's array.  The
// runtime's own pageable copy moves 23 GB/s on one thread, which also takes the page faults
// of a fresh array; the copy engine moves 211 GB/s.  Belongs to one handle; the first large
// copy makes it, on the handle's device.  The caller's current device is the same after it.
class HostStage {
  public:
    ~HostStage() { release(); }
    cudaError_t copy(void* dst, const void* src, size_t bytes, int device) {
        std::lock_guard<std::mutex> g(mu_);
        int callers = device;
        cudaError_t e = cudaGetDevice(&callers);
        if (e == cudaSuccess && callers != device) e = cudaSetDevice(device);
        if (e != cudaSuccess) return e;
        e = copy_here(dst, src, bytes, device);
        if (callers != device) {
            const cudaError_t back = cudaSetDevice(callers);
            if (e == cudaSuccess) e = back;
        }
        return e;
    }

  private:
    static constexpr int kThreads = 8;
    static constexpr size_t kChunk = size_t(1) << 20;
    // With `device` current, which the last share, done by this thread, leaves so.
    cudaError_t copy_here(void* dst, const void* src, size_t bytes, int device) {
        cudaPointerAttributes at{};
        const bool pageable = cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
        cudaGetLastError();
        if (!pageable || bytes < 4 * kChunk || !ready()) return cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost);
        cudaError_t e = cudaStreamSynchronize(nullptr);  // a copy waits for the legacy stream's work
        if (e != cudaSuccess) return e;
        std::atomic<int> failed{(int)cudaSuccess};
        auto work = [&](int t) {
            cudaError_t w = cudaSetDevice(device);
            const size_t chunks = (bytes + kChunk - 1) / kChunk;
            auto size_of = [&](size_t c) { return std::min(kChunk, bytes - c * kChunk); };
            auto fetch = [&](size_t c, int k) {
                if (w == cudaSuccess)
                    w = cudaMemcpyAsync(buf_ + (2 * t + k) * kChunk, static_cast<const char*>(src) + c * kChunk, size_of(c),
                                        cudaMemcpyDeviceToHost, stream_[t]);
                if (w == cudaSuccess) w = cudaEventRecord(event_[2 * t + k], stream_[t]);
            };
            size_t c = t;
            if (c < chunks) fetch(c, 0);
            for (int k = 0; c < chunks && w == cudaSuccess; c += kThreads, k ^= 1) {
                if (c + kThreads < chunks) fetch(c + kThreads, k ^ 1);
                if (w == cudaSuccess) w = cudaEventSynchronize(event_[2 * t + k]);
                if (w == cudaSuccess)
                    std::memcpy(static_cast<char*>(dst) + c * kChunk, buf_ + (2 * t + k) * kChunk, size_of(c));
            }
            cudaStreamSynchronize(stream_[t]);  // nothing in flight into the buffers after a failure
            if (w != cudaSuccess) failed = (int)w;
        };
        std::thread threads[kThreads];
        int started = 0;
        try {
            for (; started < kThreads - 1; ++started) threads[started] = std::thread(work, started);
        } catch (...) {  // no more threads: their shares are done here
        }
        for (int t = started; t < kThreads; ++t) work(t);
        for (int t = 0; t < started; ++t) threads[t].join();
        return (cudaError_t)failed.load();
    }

    bool ready() {
        if (buf_) return true;
        bool ok = cudaMallocHost((void**)&buf_, 2 * kThreads * kChunk) == cudaSuccess;
        for (int t = 0; t < kThreads && ok; ++t)
            ok = cudaStreamCreateWithFlags(&stream_[t], cudaStreamNonBlocking) == cudaSuccess;
        for (int k = 0; k < 2 * kThreads && ok; ++k)
            ok = cudaEventCreateWithFlags(&event_[k], cudaEventDisableTiming) == cudaSuccess;
        if (!ok) release();
        return ok;
    }
    void release() {
        for (cudaEvent_t& e : event_)
            if (e) cudaEventDestroy(e), e = nullptr;
        for (cudaStream_t& s : stream_)
            if (s) cudaStreamDestroy(s), s = nullptr;
        if (buf_) cudaFreeHost(buf_);
        buf_ = nullptr;
        cudaGetLastError();
    }
    std::mutex mu_;
    char* buf_ = nullptr;
    cudaStream_t stream_[kThreads] = {};
    cudaEvent_t event_[2 * kThreads] = {};
};
}  // namespace rs
