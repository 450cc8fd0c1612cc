// The two runtime functions of opt_in_threads.cu: setting the limit waits until both
// threads are in it, and the larger size is set first.
#include <cuda_runtime_api.h>

#include <chrono>
#include <condition_variable>
#include <mutex>

namespace {
std::mutex mu;
std::condition_variable cv;
int inside = 0;
bool larger_set = false;
}  // namespace
thread_local bool is_larger = false;
int limit = 0;

extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}

extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute attr, int value) {
    if (attr != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    std::unique_lock<std::mutex> lock(mu);
    ++inside;
    cv.notify_all();
    // both threads are here together, unless opt_in lets one in at a time
    cv.wait_for(lock, std::chrono::milliseconds(500), [] { return inside >= 2; });
    if (is_larger) {
        limit = value;
        larger_set = true;
        cv.notify_all();
    } else {
        cv.wait_for(lock, std::chrono::milliseconds(500), [] { return larger_set; });
        limit = value;
    }
    return cudaSuccess;
}
