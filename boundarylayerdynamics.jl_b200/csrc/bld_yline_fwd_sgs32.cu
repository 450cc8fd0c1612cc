// Forward line y passes: Smagorinsky spaces, single precision.
#include "bld_yline_launch.cuh"

namespace bld_yl {
cudaError_t init_fwd_sgs32() { return bld_util::init_tables(); }
cudaError_t launch_fwd_sgs32(const FwdYArgs& a, int nm, cudaStream_t st) {
    switch (a.P2) {
#define X(N) case N: return launch_fwd_p<float, N, true>(a, nm, st);
        BLD_ROW_SGS_SIZES(X)
#undef X
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace bld_yl
