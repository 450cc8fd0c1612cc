// Advection x-pass family, single precision.
#include "bld_family_adv.cuh"

namespace bld {
template int launch_adv_family<float>(bld_handle*, const Space&, const XArgs&, int);
template int setup_adv<float>();
template cudaError_t wait_limit_adv<float>(long long);
}  // namespace bld
