// In-place x kernels: Smagorinsky model, double precision.
#include "bld_xrow_launch.cuh"

namespace bld_row {
cudaError_t init_sgs64() { return init_tables(); }
cudaError_t launch_sgs64(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    return launch_sgs<double>(a, nchunks, nm, st);
}
}  // namespace bld_row
