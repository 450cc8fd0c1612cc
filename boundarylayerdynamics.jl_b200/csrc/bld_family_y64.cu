// y-pass family, double precision.
#include "bld_family_y.cuh"

namespace bld {
template int launch_inv_y<double>(bld_handle*, const Space&, InvYArgs, int);
template int launch_fwd_y<double>(bld_handle*, const Space&, FwdYArgs, int);
template int setup_y<double>();
template cudaError_t wait_limit_y<double>(long long);
}  // namespace bld
