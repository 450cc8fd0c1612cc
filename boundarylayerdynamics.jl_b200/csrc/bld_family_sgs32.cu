// Smagorinsky x-pass family, single precision.
#include "bld_family_sgs.cuh"

namespace bld {
template int launch_sgs_x<float>(bld_handle*, const Space&, const XArgs&, int);
template int setup_sgs<float>();
template cudaError_t wait_limit_sgs<float>(long long);
}  // namespace bld
