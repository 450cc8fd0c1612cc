// The Smagorinsky x passes other than the in-place one: launches and shared-memory limits.
#pragma once

#include "bld_engine.h"

namespace bld {

#define BLD_XR_CASES(KERNEL)                                                                          \
    case 2: KERNEL<R, xr_ppt(2), 2><<<grid, thr, sm, h->stream>>>(a); break;                         \
    case 3: KERNEL<R, xr_ppt(3), 3><<<grid, thr, sm, h->stream>>>(a); break;                         \
    case 4: KERNEL<R, xr_ppt(4), 4><<<grid, thr, sm, h->stream>>>(a); break;                         \
    case 6: KERNEL<R, xr_ppt(6), 6><<<grid, thr, sm, h->stream>>>(a); break;                         \
    case 8: KERNEL<R, xr_ppt(8), 8><<<grid, thr, sm, h->stream>>>(a); break;                         \
    case 9: KERNEL<R, xr_ppt(9), 9><<<grid, thr, sm, h->stream>>>(a); break;                         \
    case 12: KERNEL<R, xr_ppt(12), 12><<<grid, thr, sm, h->stream>>>(a); break;                      \
    case 16: KERNEL<R, xr_ppt(16), 16><<<grid, thr, sm, h->stream>>>(a); break;                      \
    case 24: KERNEL<R, xr_ppt(24), 24><<<grid, thr, sm, h->stream>>>(a); break;

template <typename R, int P>
int launch_sgs_x2_p(bld_handle* h, const Space& s, const XArgs& a, dim3 grid, int thr, size_t sm) {
    if constexpr (sizeof(R) == 4 && sx2_capped_size(P)) {
        if (s.sx2 == 2 || s.sx2 == 4) {
            if (s.PPT == 1)
                k_sgs_x<R, 1, 0, P, 2><<<grid, thr, sm, h->stream>>>(a);
            else
                k_sgs_x<R, 2, 0, P, 2><<<grid, thr, sm, h->stream>>>(a);
            return BLD_OK;
        }
    }
    if (s.PPT == 1)
        k_sgs_x<R, 1, 0, P><<<grid, thr, sm, h->stream>>>(a);
    else
        k_sgs_x<R, 2, 0, P><<<grid, thr, sm, h->stream>>>(a);
    return BLD_OK;
}

template <typename R, int P, int V>
void launch_sgs_xk_pv(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    constexpr int A = y2_radix_a(P), B = y2_radix_b(P);
    constexpr int NR = sx2_rows((int)sizeof(cplx<R>), P, V);
    dim3 grid(s.P2 / NR, s.nchunks, nm);
    const size_t sm = sx2_smem(A, B, h->g.K1, (int)sizeof(cplx<R>), V);
    k_sgs_x2<R, A, B, V><<<grid, sx2_threads(B, NR), sm, h->stream>>>(a);
}

template <typename R, int P>
int launch_sgs_xk_p(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    if constexpr (sizeof(R) == 4 && P <= 384) {
        if (s.sxk == 2) return launch_sgs_xk_pv<R, P, 1>(h, s, a, nm), BLD_OK;
    }
    launch_sgs_xk_pv<R, P, 0>(h, s, a, nm);
    return BLD_OK;
}

template <typename R>
int launch_sgs_xk(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    switch (s.P1) {
        case 64: BLD_TRY((launch_sgs_xk_p<R, 64>(h, s, a, nm))); break;
        case 96: BLD_TRY((launch_sgs_xk_p<R, 96>(h, s, a, nm))); break;
        case 128: BLD_TRY((launch_sgs_xk_p<R, 128>(h, s, a, nm))); break;
        case 144: BLD_TRY((launch_sgs_xk_p<R, 144>(h, s, a, nm))); break;
        case 192: BLD_TRY((launch_sgs_xk_p<R, 192>(h, s, a, nm))); break;
        case 256: BLD_TRY((launch_sgs_xk_p<R, 256>(h, s, a, nm))); break;
        case 288: BLD_TRY((launch_sgs_xk_p<R, 288>(h, s, a, nm))); break;
        default:
            if constexpr (sizeof(R) == 4) {
                if (s.P1 == 384) { BLD_TRY((launch_sgs_xk_p<R, 384>(h, s, a, nm))); break; }
                if (s.P1 == 512) { BLD_TRY((launch_sgs_xk_p<R, 512>(h, s, a, nm))); break; }
                if (s.P1 == 768) { BLD_TRY((launch_sgs_xk_p<R, 768>(h, s, a, nm))); break; }
            }
            return fail(BLD_ERR_INVALID_CONFIG, "no k_sgs_x2 kernel for P1=%d", s.P1);
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}

template <typename R>
int launch_sgs_x(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    if (s.sxk) return launch_sgs_xk<R>(h, s, a, nm);
    dim3 grid(s.P2 / s.YT, s.nchunks, nm);
    const int thr = s.YT * s.P1 / s.PPT;
    const size_t sm = smem_sgs(s, sizeof(R) == 4, h->g.K1);
    if (s.sx2) {
        switch (s.P1) {
            case 64: BLD_TRY((launch_sgs_x2_p<R, 64>(h, s, a, grid, thr, sm))); break;
            case 96: BLD_TRY((launch_sgs_x2_p<R, 96>(h, s, a, grid, thr, sm))); break;
            case 128: BLD_TRY((launch_sgs_x2_p<R, 128>(h, s, a, grid, thr, sm))); break;
            case 144: BLD_TRY((launch_sgs_x2_p<R, 144>(h, s, a, grid, thr, sm))); break;
            case 192: BLD_TRY((launch_sgs_x2_p<R, 192>(h, s, a, grid, thr, sm))); break;
            case 256: BLD_TRY((launch_sgs_x2_p<R, 256>(h, s, a, grid, thr, sm))); break;
            case 288: BLD_TRY((launch_sgs_x2_p<R, 288>(h, s, a, grid, thr, sm))); break;
            default:
                if constexpr (sizeof(R) == 4) {
                    if (s.P1 == 384) { BLD_TRY((launch_sgs_x2_p<R, 384>(h, s, a, grid, thr, sm))); break; }
                    if (s.P1 == 512) { BLD_TRY((launch_sgs_x2_p<R, 512>(h, s, a, grid, thr, sm))); break; }
                    if (s.P1 == 768) { BLD_TRY((launch_sgs_x2_p<R, 768>(h, s, a, grid, thr, sm))); break; }
                }
                return fail(BLD_ERR_INVALID_CONFIG, "no two-pass SGS x kernel for P1=%d", s.P1);
        }
        CUDA_TRY(cudaGetLastError());
        return BLD_OK;
    }
    if (s.xr) {
        switch (s.xr) {
            BLD_XR_CASES(k_sgs_x)
            default: return fail(BLD_ERR_INVALID_CONFIG, "no warp x transform of radix %d", s.xr);
        }
    } else {
        switch (s.PPT) {
            case 1: k_sgs_x<R, 1, 0><<<grid, thr, sm, h->stream>>>(a); break;
            case 2: k_sgs_x<R, 2, 0><<<grid, thr, sm, h->stream>>>(a); break;
            case 3: k_sgs_x<R, 3, 0><<<grid, thr, sm, h->stream>>>(a); break;
            default: k_sgs_x<R, 4, 0><<<grid, thr, sm, h->stream>>>(a); break;
        }
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}


template <typename R>
int setup_sgs() {
    BLD_TRY(upload_codelet_tables());
#define BLD_SET_SX2(P) BLD_SET((k_sgs_x<R, 1, 0, P>)); BLD_SET((k_sgs_x<R, 2, 0, P>));   \
    if constexpr (P <= 288) BLD_SET((k_sgs_x2<R, y2_radix_a(P), y2_radix_b(P)>));          \
    if constexpr (sizeof(R) == 4 && P <= 384) BLD_SET((k_sgs_x2<R, y2_radix_a(P), y2_radix_b(P), 1>));
    BLD_SET_SX2(64)
    BLD_SET_SX2(96)
    BLD_SET_SX2(128)
    BLD_SET_SX2(144)
    BLD_SET_SX2(192)
    BLD_SET_SX2(256)
    BLD_SET_SX2(288)
    if constexpr (sizeof(R) == 4) {
        BLD_SET_SX2(384)
        BLD_SET_SX2(512)
        BLD_SET_SX2(768)
        BLD_SET((k_sgs_x2<R, y2_radix_a(384), y2_radix_b(384)>));
        BLD_SET((k_sgs_x2<R, y2_radix_a(512), y2_radix_b(512)>));
        BLD_SET((k_sgs_x2<R, y2_radix_a(768), y2_radix_b(768)>));
#define BLD_SET_SX2C(P) BLD_SET((k_sgs_x<R, 1, 0, P, 2>)); BLD_SET((k_sgs_x<R, 2, 0, P, 2>));
        BLD_SET_SX2C(256)
        BLD_SET_SX2C(288)
        BLD_SET_SX2C(384)
        BLD_SET_SX2C(512)
        BLD_SET_SX2C(768)
#undef BLD_SET_SX2C
    }
#undef BLD_SET_SX2
    BLD_SET((k_sgs_x<R, 1, 0>));
    BLD_SET((k_sgs_x<R, 2, 0>));
    BLD_SET((k_sgs_x<R, 3, 0>));
    BLD_SET((k_sgs_x<R, 4, 0>));
#define BLD_SET_XR(r) BLD_SET((k_sgs_x<R, xr_ppt(r), r>));
    BLD_SET_XR(2)
    BLD_SET_XR(3)
    BLD_SET_XR(4)
    BLD_SET_XR(6)
    BLD_SET_XR(8)
    BLD_SET_XR(9)
    BLD_SET_XR(12)
    BLD_SET_XR(16)
    BLD_SET_XR(24)
#undef BLD_SET_XR
    return BLD_OK;
}

template <typename R>
cudaError_t wait_limit_sgs(long long cycles) {
    return cudaMemcpyToSymbol(g_bld_wait_limit, &cycles, sizeof(cycles));
}

}  // namespace bld
