// Copies between pageable host memory and the device through pinned staging buffers
// filled and emptied by a few threads.
//
// The driver stages pageable copies through one thread: 8.4 MB (one physical field at
// 128^2 x 64) take 0.79 ms up and 0.47 ms down, 3.6 ms down into memory that has not
// been touched yet.  Four threads, each with two 512 KB buffers and its own part of the
// array, take 0.40, 0.39 and 0.95 ms.  Copies under 2 MB and pinned or managed host
// memory go to the driver as they are.
//
// The buffers (4 MB) are one set per process, allocated by the first copy that needs
// them and freed with the last handle; a copy that finds them in use by another thread
// takes the driver's path.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace bld {

class HostCopy {
  public:
    static HostCopy& get() {
        static HostCopy* c = new HostCopy();   // never destroyed: handles may outlive static objects
        return *c;
    }
    void add_user() {
        std::lock_guard<std::mutex> lock(mu_);
        ++users_;
    }
    void drop_user() {
        std::lock_guard<std::mutex> lock(mu_);
        if (--users_ == 0 && pin_) {
            cudaFreeHost(pin_);
            pin_ = nullptr;
        }
    }
    // dev <- host or host <- dev, ordered on `st` of `device` (the current device).  A
    // staged copy has read or written the whole host array when this returns, a copy that
    // the driver was given may not have (from pinned memory it has only been enqueued), so
    // the caller synchronises the stream before it gives the array back.
    cudaError_t copy(void* dst, const void* src, size_t bytes, bool to_device, cudaStream_t st, int device) {
        const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
        cudaPointerAttributes at{};
        if (bytes < 4 * kChunk ||
            cudaPointerGetAttributes(&at, to_device ? src : static_cast<const void*>(dst)) != cudaSuccess ||
            at.type != cudaMemoryTypeUnregistered)
            return cudaMemcpyAsync(dst, src, bytes, kind, st);
        std::unique_lock<std::mutex> lock(mu_, std::try_to_lock);
        if (!lock.owns_lock()) return cudaMemcpyAsync(dst, src, bytes, kind, st);
        if (!pin_ && cudaHostAlloc(reinterpret_cast<void**>(&pin_), kThreads * 2 * kChunk, cudaHostAllocPortable) !=
                         cudaSuccess) {
            pin_ = nullptr;
            cudaGetLastError();
            return cudaMemcpyAsync(dst, src, bytes, kind, st);
        }
        const int parts = (int)std::min<size_t>(kThreads, bytes / kChunk);
        cudaError_t err[kThreads] = {};
        auto part = [&](int k) noexcept {
            const size_t lo = bytes / parts * k, hi = k == parts - 1 ? bytes : bytes / parts * (k + 1);
            char* pin = pin_ + (size_t)2 * kChunk * k;
            err[k] = to_device ? up(static_cast<char*>(dst) + lo, static_cast<const char*>(src) + lo, hi - lo, pin, st, device)
                               : down(static_cast<char*>(dst) + lo, static_cast<const char*>(src) + lo, hi - lo, pin, st, device);
        };
        std::thread threads[kThreads];
        int started = 1;
        try {
            for (; started < parts; ++started) threads[started] = std::thread(part, started);
        } catch (...) {   // no thread, or no memory for one: the rest here
        }
        part(0);
        for (int k = started; k < parts; ++k) part(k);
        for (int k = 1; k < started; ++k) threads[k].join();
        for (cudaError_t e : err)
            if (e != cudaSuccess) return e;
        return cudaSuccess;
    }

  private:
    static constexpr size_t kChunk = (size_t)512 << 10;
    static constexpr int kThreads = 4;
    std::mutex mu_;
    int users_ = 0;
    char* pin_ = nullptr;   // [threads][2][chunk]

    struct Events {
        cudaEvent_t ev[2] = {nullptr, nullptr};
        cudaError_t make(int device) {
            cudaError_t e = cudaSetDevice(device);
            for (auto& v : ev)
                if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
            return e;
        }
        ~Events() {
            for (auto v : ev)
                if (v) cudaEventDestroy(v);
        }
    };
    static cudaError_t up(char* dev, const char* host, size_t n, char* pin, cudaStream_t st, int device) noexcept {
        Events v;
        cudaError_t e = v.make(device);
        int i = 0;
        for (size_t o = 0; o < n && e == cudaSuccess; o += kChunk, ++i) {
            const size_t m = std::min(kChunk, n - o);
            char* p = pin + (i & 1) * kChunk;
            if (i >= 2) e = cudaEventSynchronize(v.ev[i & 1]);
            if (e != cudaSuccess) break;
            memcpy(p, host + o, m);
            e = cudaMemcpyAsync(dev + o, p, m, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(v.ev[i & 1], st);
        }
        // the buffers are reused after the return
        for (int k = 0; k < std::min(i, 2); ++k) {
            const cudaError_t w = cudaEventSynchronize(v.ev[k]);
            if (e == cudaSuccess) e = w;
        }
        return e;
    }
    static cudaError_t down(char* host, const char* dev, size_t n, char* pin, cudaStream_t st, int device) noexcept {
        Events v;
        cudaError_t e = v.make(device);
        const size_t chunks = (n + kChunk - 1) / kChunk;
        for (size_t c = 0; c <= chunks && e == cudaSuccess; ++c) {
            if (c < chunks) {
                const size_t o = c * kChunk;
                e = cudaMemcpyAsync(pin + (c & 1) * kChunk, dev + o, std::min(kChunk, n - o), cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaEventRecord(v.ev[c & 1], st);
            }
            if (c > 0 && e == cudaSuccess) {
                const size_t o = (c - 1) * kChunk;
                e = cudaEventSynchronize(v.ev[(c - 1) & 1]);
                if (e == cudaSuccess) memcpy(host + o, pin + ((c - 1) & 1) * kChunk, std::min(kChunk, n - o));
            }
        }
        if (e != cudaSuccess) cudaStreamSynchronize(st);   // nothing may still write the buffers
        return e;
    }
};

}  // namespace bld
