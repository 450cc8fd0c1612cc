// y-pass family, single precision.
#include "bld_family_y.cuh"

namespace bld {
template int launch_inv_y<float>(bld_handle*, const Space&, InvYArgs, int);
template int launch_fwd_y<float>(bld_handle*, const Space&, FwdYArgs, int);
template int setup_y<float>();
template cudaError_t wait_limit_y<float>(long long);
}  // namespace bld
