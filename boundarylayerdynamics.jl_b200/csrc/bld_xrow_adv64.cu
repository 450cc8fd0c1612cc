// In-place x kernels: advection, double precision.
#include "bld_xrow_launch.cuh"

namespace bld_row {
cudaError_t init_adv64() { return init_tables(); }
cudaError_t launch_adv64(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    return launch_adv<double>(a, nchunks, nm, st);
}
}  // namespace bld_row
