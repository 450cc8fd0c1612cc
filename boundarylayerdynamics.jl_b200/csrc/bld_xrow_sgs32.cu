// In-place x kernels: Smagorinsky model, single precision.
#include "bld_xrow_launch.cuh"

namespace bld_row {
cudaError_t init_sgs32() { return init_tables(); }
cudaError_t launch_sgs32(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    return launch_sgs<float>(a, nchunks, nm, st);
}
}  // namespace bld_row
