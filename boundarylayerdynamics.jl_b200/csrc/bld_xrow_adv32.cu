// In-place x kernels: advection, single precision.
#include "bld_xrow_launch.cuh"

namespace bld_row {
cudaError_t init_adv32() { return init_tables(); }
cudaError_t launch_adv32(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    return launch_adv<float>(a, nchunks, nm, st);
}
}  // namespace bld_row
