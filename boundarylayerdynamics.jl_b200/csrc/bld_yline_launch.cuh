// Launchers of the line y passes; each translation unit instantiates one of them.
#pragma once

#include "bld_launch_util.cuh"
#include "bld_yline.h"
#include "bld_ylines.cuh"

namespace bld_yl {

// band: 1 with the 3/2 rule where the pruned radix is a multiple of 3, 2 on the default grid
template <typename R, int P, bool SGS>
cudaError_t launch_inv_p(InvYArgs a, int nm, cudaStream_t st) {
    constexpr Shape s = inv_shape(P, sizeof(R) == 4, SGS);
    if constexpr (s.A > 0) {
        static std::atomic<int> done[64];
        const auto k = k_inv_yl<R, s.A, s.B, s.NL, s.MINB, SGS ? 2 : (s.A % 3 == 0 ? 1 : 0), SGS>;
        const int sm = smem_bytes(s.A, s.B, s.NL, (int)sizeof(cplx<R>), 1);
        if (const cudaError_t e = bld_util::opt_in(k, sm, done); e != cudaSuccess) return e;
        a.NL = s.NL;
        return bld_util::launch(k, dim3(a.nterms * nm, (a.g.K1 + s.NL - 1) / s.NL, a.g.n3),
                                (s.A > s.B ? s.A : s.B) * s.NL, sm, st, a.overlap != 0, a);
    }
    return cudaErrorInvalidValue;
}

template <typename R, int P, bool SGS>
cudaError_t launch_fwd_p(FwdYArgs a, int nm, cudaStream_t st) {
    constexpr Shape s = fwd_shape(P, sizeof(R) == 4, SGS);
    if constexpr (s.A > 0) {
        static std::atomic<int> done[64];
        const auto k = k_fwd_yl<R, s.A, s.B, s.NL, s.MINB, SGS ? 2 : (s.B % 3 == 0 ? 1 : 0), SGS ? 2 : 1>;
        const int sm = smem_bytes(s.A, s.B, s.NL, (int)sizeof(cplx<R>), SGS ? 2 : 1);
        if (const cudaError_t e = bld_util::opt_in(k, sm, done); e != cudaSuccess) return e;
        a.NL = s.NL;
        return bld_util::launch(k, dim3(a.fields * nm, (a.g.K1 + s.NL - 1) / s.NL, a.g.n3),
                                (s.A > s.B ? s.A : s.B) * s.NL, sm, st, a.overlap != 0, a);
    }
    return cudaErrorInvalidValue;
}

}  // namespace bld_yl
