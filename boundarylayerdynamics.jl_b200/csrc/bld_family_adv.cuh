// The advection x passes other than the in-place one: launches and shared-memory limits.
#pragma once

#include "bld_engine.h"

namespace bld {

template <typename R, int P, int V>
void launch_x2_pv(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    constexpr int A = y2_radix_a(P), B = y2_radix_b(P);
    constexpr int NR = x2_rows((int)sizeof(cplx<R>), P, V);
    dim3 grid(s.P2 / NR, s.nchunks, nm);
    const size_t sm = x2_smem(A, B, h->g.K1, (int)sizeof(cplx<R>), V);
    k_adv_x2<R, A, B, V><<<grid, x2_threads(B, NR, V), sm, h->stream>>>(a, h->flag);
}

template <typename R, int P>
int launch_x2_p(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    if constexpr (sizeof(R) == 8) {
        if (s.x2 == 3) return launch_x2_pv<R, P, 2>(h, s, a, nm), BLD_OK;
    }
    if constexpr (sizeof(R) == 4 && P <= 384) {
        if (s.x2 == 4) return launch_x2_pv<R, P, 3>(h, s, a, nm), BLD_OK;
    }
    launch_x2_pv<R, P, 0>(h, s, a, nm);
    return BLD_OK;
}

template <typename R>
int launch_adv_x2(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    switch (s.P1) {
        case 64: BLD_TRY((launch_x2_p<R, 64>(h, s, a, nm))); break;
        case 96: BLD_TRY((launch_x2_p<R, 96>(h, s, a, nm))); break;
        case 128: BLD_TRY((launch_x2_p<R, 128>(h, s, a, nm))); break;
        case 144: BLD_TRY((launch_x2_p<R, 144>(h, s, a, nm))); break;
        case 192: BLD_TRY((launch_x2_p<R, 192>(h, s, a, nm))); break;
        case 256: BLD_TRY((launch_x2_p<R, 256>(h, s, a, nm))); break;
        case 288: BLD_TRY((launch_x2_p<R, 288>(h, s, a, nm))); break;
        default:
            if constexpr (sizeof(R) == 4) {
                if (s.P1 == 384) { BLD_TRY((launch_x2_p<R, 384>(h, s, a, nm))); break; }
                if (s.P1 == 512) { BLD_TRY((launch_x2_p<R, 512>(h, s, a, nm))); break; }
                if (s.P1 == 768) { BLD_TRY((launch_x2_p<R, 768>(h, s, a, nm))); break; }
            }
            return fail(BLD_ERR_INVALID_CONFIG, "no two-pass x kernel for P1=%d", s.P1);
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}

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

template <typename R>
int launch_adv_x(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    dim3 grid(s.P2 / s.YT, s.nchunks, nm);
    const int thr = s.YT * s.P1 / s.PPT;
    const size_t sm = smem_adv(s, sizeof(R) == 4);
    if (s.xr) {
        switch (s.xr) {
            BLD_XR_CASES(k_adv_x)
            default: return fail(BLD_ERR_INVALID_CONFIG, "no warp x transform of radix %d", s.xr);
        }
    } else {
        switch (s.PPT) {
            case 1: k_adv_x<R, 1, 0><<<grid, thr, sm, h->stream>>>(a); break;
            case 2: k_adv_x<R, 2, 0><<<grid, thr, sm, h->stream>>>(a); break;
            case 3: k_adv_x<R, 3, 0><<<grid, thr, sm, h->stream>>>(a); break;
            default: k_adv_x<R, 4, 0><<<grid, thr, sm, h->stream>>>(a); break;
        }
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}

template <typename R>
int launch_adv_xw(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    const int r = warpx_radix<R>(s.P1);
    dim3 grid((s.P2 + s.xw - 1) / s.xw, s.nchunks, nm);
    const int thr = 32 * s.xw;
    const size_t sm = ((size_t)r * 32 + (size_t)s.xw * 12 * h->g.K1) * csize(sizeof(R) == 4);
    if constexpr (sizeof(R) == 4) {
        if (s.xwmb > 1) {
            if (!warpx_minb_ok<R>(r, s.xwmb)) return fail(BLD_ERR_INVALID_CONFIG, "no capped warp x kernel");
#define BLD_XW_MB(RR)                                                                   \
    case RR:                                                                            \
        if (s.xwmb == 3) k_adv_xwc<R, RR, 3><<<grid, thr, sm, h->stream>>>(a);          \
        else k_adv_xwc<R, RR, 4><<<grid, thr, sm, h->stream>>>(a);                      \
        break;
            switch (r) {
                BLD_XW_MB(8)
                BLD_XW_MB(9)
                BLD_XW_MB(12)
                default: return fail(BLD_ERR_INVALID_CONFIG, "no capped warp x kernel");
            }
#undef BLD_XW_MB
            CUDA_TRY(cudaGetLastError());
            return BLD_OK;
        }
    }
    switch (r) {
        case 2: k_adv_xw<R, 2><<<grid, thr, sm, h->stream>>>(a); break;
        case 3: k_adv_xw<R, 3><<<grid, thr, sm, h->stream>>>(a); break;
        case 4: k_adv_xw<R, 4><<<grid, thr, sm, h->stream>>>(a); break;
        case 6: k_adv_xw<R, 6><<<grid, thr, sm, h->stream>>>(a); break;
        default:
            if constexpr (sizeof(R) == 4) {
                switch (r) {
                    case 8: k_adv_xw<R, 8><<<grid, thr, sm, h->stream>>>(a); break;
                    case 9: k_adv_xw<R, 9><<<grid, thr, sm, h->stream>>>(a); break;
                    case 12: k_adv_xw<R, 12><<<grid, thr, sm, h->stream>>>(a); break;
                    default: return fail(BLD_ERR_INVALID_CONFIG, "no warp x kernel for P1=%d", s.P1);
                }
            } else {
                return fail(BLD_ERR_INVALID_CONFIG, "no warp x kernel for P1=%d", s.P1);
            }
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}

template <typename R>
int launch_adv_xb(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    const int r = xb_radix(s.P1, sizeof(R) == 4);
    dim3 grid(s.P2, s.nchunks, nm);
    if (s.xb == 2) {
        const size_t smp = ((size_t)r * 32 + 5 * (size_t)(s.P1 + 32) + 12 * (size_t)h->g.K1) * csize(sizeof(R) == 4);
        switch (r) {
            case 2: k_adv_xp<R, 2><<<grid, 160, smp, h->stream>>>(a); break;
            case 3: k_adv_xp<R, 3><<<grid, 160, smp, h->stream>>>(a); break;
            case 4: k_adv_xp<R, 4><<<grid, 160, smp, h->stream>>>(a); break;
            case 6: k_adv_xp<R, 6><<<grid, 160, smp, h->stream>>>(a); break;
            case 8: k_adv_xp<R, 8><<<grid, 160, smp, h->stream>>>(a); break;
            case 9: k_adv_xp<R, 9><<<grid, 160, smp, h->stream>>>(a); break;
            case 12: k_adv_xp<R, 12><<<grid, 160, smp, h->stream>>>(a); break;
            default:
                if constexpr (sizeof(R) == 4) {
                    if (r == 16) { k_adv_xp<R, 16><<<grid, 160, smp, h->stream>>>(a); break; }
                    if (r == 24) { k_adv_xp<R, 24><<<grid, 160, smp, h->stream>>>(a); break; }
                }
                return fail(BLD_ERR_INVALID_CONFIG, "no pipelined block-of-warps x kernel for P1=%d", s.P1);
        }
        CUDA_TRY(cudaGetLastError());
        return BLD_OK;
    }
    const size_t sm = ((size_t)r * 32 + 3 * (size_t)(s.P1 + 32) + 12 * (size_t)h->g.K1) * csize(sizeof(R) == 4);
    switch (r) {
        case 2: k_adv_xb<R, 2><<<grid, 96, sm, h->stream>>>(a); break;
        case 3: k_adv_xb<R, 3><<<grid, 96, sm, h->stream>>>(a); break;
        case 4: k_adv_xb<R, 4><<<grid, 96, sm, h->stream>>>(a); break;
        case 6: k_adv_xb<R, 6><<<grid, 96, sm, h->stream>>>(a); break;
        case 8: k_adv_xb<R, 8><<<grid, 96, sm, h->stream>>>(a); break;
        case 9: k_adv_xb<R, 9><<<grid, 96, sm, h->stream>>>(a); break;
        case 12: k_adv_xb<R, 12><<<grid, 96, sm, h->stream>>>(a); break;
        default:
            if constexpr (sizeof(R) == 4) {
                if (r == 16) { k_adv_xb<R, 16><<<grid, 96, sm, h->stream>>>(a); break; }
                if (r == 24) { k_adv_xb<R, 24><<<grid, 96, sm, h->stream>>>(a); break; }
            }
            return fail(BLD_ERR_INVALID_CONFIG, "no block-of-warps x kernel for P1=%d", s.P1);
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}

// the family the autotuner (or a switch) chose
template <typename R>
int launch_adv_family(bld_handle* h, const Space& s, const XArgs& a, int nm) {
    if (s.x2) return launch_adv_x2<R>(h, s, a, nm);
    if (s.xb) return launch_adv_xb<R>(h, s, a, nm);
    return s.xw ? launch_adv_xw<R>(h, s, a, nm) : launch_adv_x<R>(h, s, a, nm);
}

template <typename R>
int setup_adv() {
    BLD_TRY(upload_codelet_tables());
#define BLD_SET_X2(P)                                                   \
    BLD_SET((k_adv_x2<R, y2_radix_a(P), y2_radix_b(P), 0>));            \
    if constexpr (sizeof(R) == 8) {                                     \
        BLD_SET((k_adv_x2<R, y2_radix_a(P), y2_radix_b(P), 2>));        \
    }                                                                   \
    if constexpr (sizeof(R) == 4 && P <= 384) {                         \
        BLD_SET((k_adv_x2<R, y2_radix_a(P), y2_radix_b(P), 3>));        \
    }
    BLD_SET_X2(64)
    BLD_SET_X2(96)
    BLD_SET_X2(128)
    BLD_SET_X2(144)
    BLD_SET_X2(192)
    BLD_SET_X2(256)
    BLD_SET_X2(288)
    if constexpr (sizeof(R) == 4) {
        BLD_SET_X2(384)
        BLD_SET_X2(512)
        BLD_SET_X2(768)
    }
#undef BLD_SET_X2
    BLD_SET((k_adv_x<R, 1, 0>));
    BLD_SET((k_adv_x<R, 2, 0>));
    BLD_SET((k_adv_x<R, 3, 0>));
    BLD_SET((k_adv_x<R, 4, 0>));
#define BLD_SET_XR(r) BLD_SET((k_adv_x<R, xr_ppt(r), r>));
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
    BLD_SET((k_adv_xb<R, 2>));
    BLD_SET((k_adv_xb<R, 3>));
    BLD_SET((k_adv_xb<R, 4>));
    BLD_SET((k_adv_xb<R, 6>));
    BLD_SET((k_adv_xb<R, 8>));
    BLD_SET((k_adv_xb<R, 9>));
    BLD_SET((k_adv_xb<R, 12>));
    BLD_SET((k_adv_xp<R, 2>));
    BLD_SET((k_adv_xp<R, 3>));
    BLD_SET((k_adv_xp<R, 4>));
    BLD_SET((k_adv_xp<R, 6>));
    BLD_SET((k_adv_xp<R, 8>));
    BLD_SET((k_adv_xp<R, 9>));
    BLD_SET((k_adv_xp<R, 12>));
    if constexpr (sizeof(R) == 4) {
        BLD_SET((k_adv_xb<R, 16>));
        BLD_SET((k_adv_xb<R, 24>));
        BLD_SET((k_adv_xp<R, 16>));
        BLD_SET((k_adv_xp<R, 24>));
    }
    BLD_SET((k_adv_xw<R, 2>));
    BLD_SET((k_adv_xw<R, 3>));
    BLD_SET((k_adv_xw<R, 4>));
    BLD_SET((k_adv_xw<R, 6>));
    if constexpr (sizeof(R) == 4) {
        BLD_SET((k_adv_xw<R, 8>));
        BLD_SET((k_adv_xw<R, 9>));
        BLD_SET((k_adv_xw<R, 12>));
        BLD_SET((k_adv_xwc<R, 8, 3>));
        BLD_SET((k_adv_xwc<R, 9, 3>));
        BLD_SET((k_adv_xwc<R, 12, 3>));
        BLD_SET((k_adv_xwc<R, 8, 4>));
        BLD_SET((k_adv_xwc<R, 9, 4>));
        BLD_SET((k_adv_xwc<R, 12, 4>));
    }
    return BLD_OK;
}

template <typename R>
cudaError_t wait_limit_adv(long long cycles) {
    return cudaMemcpyToSymbol(g_bld_wait_limit, &cycles, sizeof(cycles));
}

}  // namespace bld
