// The block Smagorinsky x kernels of the sizes above the in-place ones' in double precision,
// for the compiler's report of their registers.
#include <cuda_runtime.h>

#include <type_traits>
#include <utility>

#include "bld.h"
#include "bld_kernels.cuh"

double2 h_wtab64[BLD_WTAB_SIZE];
float2 h_wtab32[BLD_WTAB_SIZE];

template __global__ void k_sgs_x<double, 4, 0>(XArgs);
template __global__ void k_sgs_x<double, 3, 0>(XArgs);
template __global__ void k_sgs_x<double, 3, 12>(XArgs);
