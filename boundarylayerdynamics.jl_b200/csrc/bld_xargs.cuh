// Grid geometry and arguments shared by the x kernels of all translation units.
#pragma once

#include "bld_fft.cuh"

struct Geo {
    int K1, K2, k1max, k2max, n3, F;  // F = K1*K2 modes per layer
    long long mstride;                // complex values per member state (3*n3-1)*F
};

__host__ __device__ __forceinline__ long long fld_off(const Geo& g, int f) { return (long long)f * g.n3 * g.F; }

// inactive ensemble slots (serving) skip their blocks; uniform per block
#define BLD_SKIP_INACTIVE(a, m) \
    if ((a).active && !(a).active[m]) return

// arguments of the physical x kernels
struct XArgs {
    Geo g;
    int P1, P2, YT, zchunk;
    int m0;
    const int* active;
    const void* min;
    void* mout;
    long long min_mstride, mout_mstride;  // elements per member
    FftPlan plan;
    const void* tw;
    // SGS only
    const double* alpha_c;   // [n3]
    const double* alpha_i;   // [n3-1]
    const double* lc;        // [members][n3]   Smagorinsky length^2 at C nodes
    const double* li;        // [members][n3-1] ... at I nodes
    const double* wall;      // [members][4]: strain factor lo, hi; stress factor lo, hi
    int dyn_lo, dyn_hi;      // rough wall (dynamic wall-model values) below / above
    double w_lo, w_hi;       // Dirichlet values of vel3
    // two-pass SGS kernel: the input rows of layer j + 1 are copied into shared
    // memory by 1-d TMA bulk copies while layer j is processed (needs YT K1
    // elements to fill whole 16-byte units); a timed-out wait sets flag[m]
    int staged;
    int* flag;
    // ceil(2^32 / K1) and ceil(2^32 / P1) (0 for a divisor of 1): fdiv
    unsigned k1_magic, p1_magic;
    // row kernels (bld_xrows.cuh): [K1] k1 * 2pi/L1, and the device's limit of bounded waits
    const double* d1;
    const long long* wait_limit;
    int overlap;   // launched overlapping the kernel before it (row kernels)
    // Smagorinsky row kernel: the power of two that a vertical stress derivative is scaled
    // by while it shares a complex line with a stress, and alpha_c, alpha_i times it
    double d3_scale;
    float d3_scale32;
    const double* d3_alpha_c;
    const double* d3_alpha_i;
};

// n / d for 0 <= n < 2^16 and 1 <= d < 2^16 by one multiply-high with
// magic = ceil(2^32 / d) (0 for d = 1): with n = q d + r, n magic / 2^32 exceeds
// n / d by less than 2^-16 <= 1 / d, so its floor is q.  Replaces runtime integer
// divisions (tens of instructions each) in the index arithmetic of the x kernels.
__host__ __device__ __forceinline__ int fdiv(int n, unsigned magic) {
#ifdef __CUDA_ARCH__
    return magic ? (int)__umulhi((unsigned)n, magic) : n;
#else
    return magic ? (int)(((unsigned long long)(unsigned)n * magic) >> 32) : n;
#endif
}
inline unsigned fdiv_magic(unsigned d) { return d <= 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }

template <typename C>
__device__ __forceinline__ const C* mrow(const C* M, const XArgs& a, int t, int z, int y) {
    return M + ((long long)(t * a.g.n3 + z) * a.P2 + y) * a.g.K1;
}
template <typename C>
__device__ __forceinline__ C* mrow_w(C* M, const XArgs& a, int t, int z, int y) {
    return M + ((long long)(t * a.g.n3 + z) * a.P2 + y) * a.g.K1;
}
