// Advection x-pass family, double precision.
#include "bld_family_adv.cuh"

namespace bld {
template int launch_adv_family<double>(bld_handle*, const Space&, const XArgs&, int);
template int setup_adv<double>();
template cudaError_t wait_limit_adv<double>(long long);
}  // namespace bld
