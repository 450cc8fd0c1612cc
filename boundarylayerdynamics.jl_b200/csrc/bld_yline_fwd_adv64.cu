// Forward line y passes: advection spaces, double precision.
#include "bld_yline_launch.cuh"

namespace bld_yl {
cudaError_t init_fwd_adv64() { return bld_util::init_tables(); }
cudaError_t launch_fwd_adv64(const FwdYArgs& a, int nm, cudaStream_t st) {
    switch (a.P2) {
#define X(N) case N: return launch_fwd_p<double, N, false>(a, nm, st);
        BLD_YL_ADV_SIZES(X)
#undef X
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace bld_yl
