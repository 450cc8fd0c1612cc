// Helpers of the translation units that hold kernels: codelet tables and opt-in to large
// dynamic shared memory.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

#include "bld_dft.cuh"

namespace bld_util {

// copies the codelet twiddles to this translation unit's tables on the current device
inline cudaError_t init_tables() {
    cudaError_t e = cudaMemcpyToSymbol(c_wtab64, h_wtab64, sizeof(h_wtab64));
    return e == cudaSuccess ? cudaMemcpyToSymbol(c_wtab32, h_wtab32, sizeof(h_wtab32)) : e;
}

// the most dynamic shared memory a B200 block may opt into
constexpr int kMaxSmem = 227 * 1024;

// Opts `kernel` in to kMaxSmem bytes of dynamic shared memory and the largest carveout on
// the current device, once per device.  The limit is the same whatever `smem` the launch
// asks for (the bytes of one instantiation depend on the grid): threads that come here at
// the same time set the same value, so none lowers a limit another one relies on.
template <typename K>
cudaError_t opt_in(K kernel, int smem, std::atomic<int> (&done)[64]) {
    if (smem > kMaxSmem) return cudaErrorInvalidValue;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && done[dev].load()) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess && dev < 64) done[dev].store(1);
    return e;
}

// launches `kernel`; with `overlap` its blocks may be set up while the last blocks of the
// kernel before it on the stream still run (they wait in grid_wait before they read
// anything)
template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool overlap, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace bld_util
