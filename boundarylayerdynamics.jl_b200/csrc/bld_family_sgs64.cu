// Smagorinsky x-pass family, double precision.
#include "bld_family_sgs.cuh"

namespace bld {
template int launch_sgs_x<double>(bld_handle*, const Space&, const XArgs&, int);
template int setup_sgs<double>();
template cudaError_t wait_limit_sgs<double>(long long);
}  // namespace bld
