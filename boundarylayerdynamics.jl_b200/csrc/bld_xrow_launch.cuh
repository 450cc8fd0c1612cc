// Launchers of the in-place x kernels; each translation unit instantiates one of them.
#pragma once

#include "bld_launch_util.cuh"
#include "bld_xrow.h"
#include "bld_xrows.cuh"

namespace bld_row {

using bld_util::init_tables;
using bld_util::opt_in;

template <typename R, int P>
cudaError_t launch_adv_p(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    constexpr Shape s = adv_shape(P, sizeof(R) == 4);
    if constexpr (s.A > 0) {
        static std::atomic<int> done[64];
        const auto k = k_adv_row<R, s.A, s.B, s.NR, s.T, s.MINB, s.sepf>;
        const int sm = ar_smem(s.A, s.B, a.g.K1, (int)sizeof(cplx<R>), s.NR, s.sepf);
        if (const cudaError_t e = opt_in(k, sm, done); e != cudaSuccess) return e;
        return bld_util::launch(k, dim3((a.P2 + s.NR - 1) / s.NR, nchunks, nm), s.T, sm, st, a.overlap != 0, a);
    }
    return cudaErrorInvalidValue;
}

template <typename R, int P>
cudaError_t launch_sgs_p(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    constexpr Shape s = sgs_shape(P, sizeof(R) == 4);
    if constexpr (s.A > 0) {
        static std::atomic<int> done[64];
        const auto k = k_sgs_x<R, s.A, s.B, s.NR, s.T, s.MINB>;
        const int sm = sr_smem(s.A, s.B, a.g.K1, (int)sizeof(cplx<R>), s.NR);
        if (const cudaError_t e = opt_in(k, sm, done); e != cudaSuccess) return e;
        return bld_util::launch(k, dim3(a.P2 / s.NR, nchunks, nm), s.T, sm, st, a.overlap != 0, a);
    }
    return cudaErrorInvalidValue;
}

template <typename R>
cudaError_t launch_adv(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    switch (a.P1) {
#define X(N) case N: return launch_adv_p<R, N>(a, nchunks, nm, st);
        BLD_ROW_ADV_SIZES(X)
#undef X
        default: return cudaErrorInvalidValue;
    }
}

template <typename R>
cudaError_t launch_sgs(const XArgs& a, int nchunks, int nm, cudaStream_t st) {
    switch (a.P1) {
#define X(N) case N: return launch_sgs_p<R, N>(a, nchunks, nm, st);
        BLD_ROW_SGS_SIZES(X)
#undef X
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bld_row
