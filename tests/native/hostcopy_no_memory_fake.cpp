// The runtime functions of bld_hostcopy.h without a device: copies are done at once.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>

extern "C" {
cudaError_t CUDARTAPI cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(dst, src, n);
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = malloc(n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t CUDARTAPI cudaFreeHost(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaSetDevice(int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetLastError() { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}
