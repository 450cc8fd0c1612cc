// The y passes: launches and shared-memory limits.
#pragma once

#include "bld_engine.h"

namespace bld {

template <typename R, int P>
int launch_y2_p(bld_handle* h, bool inverse, const void* args, dim3 grid, size_t sm, int tp) {
    constexpr int A = y2_radix_a(P), B = y2_radix_b(P);
    constexpr int MINB = y2_min_blocks<R>(B * BLD_Y2_NL);
    constexpr int MINBI = y2_min_blocks_inv<R>(B * BLD_Y2_NL);
    if (!inverse && tp == 3)
        k_fwd_y2<R, A, B, 3, 8, 4><<<grid, B * 8, sm, h->stream>>>(*static_cast<const FwdYArgs*>(args));
    else if (inverse && tp == 3)   // eight lines: three (double) or four (single precision) blocks per SM
        k_inv_y2<R, A, B, sizeof(R) == 8 ? 3 : 4, 8><<<grid, B * 8, sm, h->stream>>>(
            *static_cast<const InvYArgs*>(args));
    else if (!inverse && tp == 4 && sizeof(R) == 4)
        k_fwd_y2<R, A, B, MINB, BLD_Y2_NL, 2><<<grid, B * BLD_Y2_NL, sm, h->stream>>>(
            *static_cast<const FwdYArgs*>(args));
    else if (inverse)
        k_inv_y2<R, A, B, MINBI><<<grid, B * BLD_Y2_NL, sm, h->stream>>>(*static_cast<const InvYArgs*>(args));
    else
        k_fwd_y2<R, A, B, MINB><<<grid, B * BLD_Y2_NL, sm, h->stream>>>(*static_cast<const FwdYArgs*>(args));
    return BLD_OK;
}

template <typename R>
int launch_y2(bld_handle* h, int P2, bool inverse, const void* args, dim3 grid, size_t sm, int tp = 1) {
    switch (P2) {
        case 64: return launch_y2_p<R, 64>(h, inverse, args, grid, sm, tp);
        case 96: return launch_y2_p<R, 96>(h, inverse, args, grid, sm, tp);
        case 128: return launch_y2_p<R, 128>(h, inverse, args, grid, sm, tp);
        case 144: return launch_y2_p<R, 144>(h, inverse, args, grid, sm, tp);
        case 192: return launch_y2_p<R, 192>(h, inverse, args, grid, sm, tp);
        case 256: return launch_y2_p<R, 256>(h, inverse, args, grid, sm, tp);
        case 288: return launch_y2_p<R, 288>(h, inverse, args, grid, sm, tp);
        default: break;
    }
    if constexpr (sizeof(R) == 4) {
        switch (P2) {
            case 384: return launch_y2_p<R, 384>(h, inverse, args, grid, sm, tp);
            case 512: return launch_y2_p<R, 512>(h, inverse, args, grid, sm, tp);
            case 768: return launch_y2_p<R, 768>(h, inverse, args, grid, sm, tp);
            default: break;
        }
    }
    return fail(BLD_ERR_INVALID_CONFIG, "no two-pass y transform for P2=%d", P2);
}

template <typename R, int P>
int launch_y3_p(bld_handle* h, const InvYArgs& a, const CUtensorMap& map, dim3 grid) {
    constexpr int A = y2_radix_a(P), B = y2_radix_b(P);
    const size_t sm = y3_smem(P, h->g.K2, (int)sizeof(cplx<R>));
    k_inv_y3<R, A, B><<<grid, B * BLD_Y3_NL, sm, h->stream>>>(a, map);
    return BLD_OK;
}

template <typename R>
int launch_inv_y3(bld_handle* h, const Space& s, InvYArgs a, int nm) {
    CUtensorMap map;
    BLD_TRY(state_tmap(h, a.state, BLD_Y3_NL, &map));
    a.NL = BLD_Y3_NL;
    a.zchunk = (h->g.n3 + s.inv.zc - 1) / s.inv.zc;
    a.flag = h->flag;
    dim3 grid(a.nterms * nm, (h->g.K1 + BLD_Y3_NL - 1) / BLD_Y3_NL, (h->g.n3 + a.zchunk - 1) / a.zchunk);
    switch (s.P2) {
        case 64: return launch_y3_p<R, 64>(h, a, map, grid);
        case 96: return launch_y3_p<R, 96>(h, a, map, grid);
        case 128: return launch_y3_p<R, 128>(h, a, map, grid);
        case 144: return launch_y3_p<R, 144>(h, a, map, grid);
        case 192: return launch_y3_p<R, 192>(h, a, map, grid);
        case 256: return launch_y3_p<R, 256>(h, a, map, grid);
        case 288: return launch_y3_p<R, 288>(h, a, map, grid);
        default: break;
    }
    if constexpr (sizeof(R) == 4) {
        switch (s.P2) {
            case 384: return launch_y3_p<R, 384>(h, a, map, grid);
            case 512: return launch_y3_p<R, 512>(h, a, map, grid);
            case 768: return launch_y3_p<R, 768>(h, a, map, grid);
            default: break;
        }
    }
    return fail(BLD_ERR_INVALID_CONFIG, "no TMA y transform for P2=%d", s.P2);
}

template <typename R>
int launch_inv_y(bld_handle* h, const Space& s, InvYArgs a, int nm) {
    const YCfg& c = s.inv;
    a.NL = c.NL;
    const size_t cs = csize(sizeof(R) == 4);
    if (c.tp == 2) {
        BLD_TRY(launch_inv_y3<R>(h, s, a, nm));
        CUDA_TRY(cudaGetLastError());
        return BLD_OK;
    }
    if (c.tp) {
        const int nl = c.tp == 3 ? 8 : BLD_Y2_NL;
        a.NL = nl;
        dim3 grid(a.nterms * nm, (h->g.K1 + nl - 1) / nl, h->g.n3);
        BLD_TRY(launch_y2<R>(h, s.P2, true, &a, grid, smem_y2(s.P2, nl, sizeof(R) == 4), c.tp));
        CUDA_TRY(cudaGetLastError());
        return BLD_OK;
    }
    if (c.all) {
        dim3 grid((h->g.K1 + c.NL - 1) / c.NL, h->g.n3, nm);
        k_inv_y_all<R><<<grid, c.thr, (size_t)(s.P2 + s.P2 * a.nterms * c.NL) * cs, h->stream>>>(a);
    } else {
        dim3 grid(a.nterms * nm, (h->g.K1 + c.NL - 1) / c.NL, h->g.n3);
        const size_t sm = smem_y_term(s.P2, c.NL, c.wfft, sizeof(R) == 4);
        switch (c.wfft) {
            case 0: k_inv_y<R, 0><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 2: k_inv_y<R, 2><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 3: k_inv_y<R, 3><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 4: k_inv_y<R, 4><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 6: k_inv_y<R, 6><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 8: k_inv_y<R, 8><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 9: k_inv_y<R, 9><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 12: k_inv_y<R, 12><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 16: k_inv_y<R, 16><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 24:
                if constexpr (sizeof(R) == 4) {
                    k_inv_y<R, 24><<<grid, c.thr, sm, h->stream>>>(a);
                    break;
                }
                return fail(BLD_ERR_INVALID_CONFIG, "no warp y transform of radix %d", c.wfft);
            default: return fail(BLD_ERR_INVALID_CONFIG, "no warp y transform of radix %d", c.wfft);
        }
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}

template <typename R>
int launch_fwd_y(bld_handle* h, const Space& s, FwdYArgs a, int nm) {
    const YCfg& c = s.fwd;
    a.NL = c.NL;
    const size_t cs = csize(sizeof(R) == 4);
    if (c.tp) {
        const int nl = c.tp == 3 ? 8 : BLD_Y2_NL;   // tp 1, 2, 4: BLD_Y2_NL lines
        a.NL = nl;
        dim3 grid(a.fields * nm, (h->g.K1 + nl - 1) / nl, h->g.n3);
        BLD_TRY(launch_y2<R>(h, s.P2, false, &a, grid, smem_y2(s.P2, s.fsets * nl, sizeof(R) == 4), c.tp));
        CUDA_TRY(cudaGetLastError());
        return BLD_OK;
    }
    if (c.all) {
        dim3 grid((h->g.K1 + c.NL - 1) / c.NL, h->g.n3, nm);
        k_fwd_y_all<R><<<grid, c.thr, (size_t)(s.P2 + s.P2 * 3 * s.fsets * c.NL) * cs, h->stream>>>(a);
    } else {
        dim3 grid(a.fields * nm, (h->g.K1 + c.NL - 1) / c.NL, h->g.n3);
        const size_t sm = smem_y_term(s.P2, s.fsets * c.NL, c.wfft, sizeof(R) == 4);
        switch (c.wfft) {
            case 0: k_fwd_y<R, 0><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 2: k_fwd_y<R, 2><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 3: k_fwd_y<R, 3><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 4: k_fwd_y<R, 4><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 6: k_fwd_y<R, 6><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 8: k_fwd_y<R, 8><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 9: k_fwd_y<R, 9><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 12: k_fwd_y<R, 12><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 16: k_fwd_y<R, 16><<<grid, c.thr, sm, h->stream>>>(a); break;
            case 24:
                if constexpr (sizeof(R) == 4) {
                    k_fwd_y<R, 24><<<grid, c.thr, sm, h->stream>>>(a);
                    break;
                }
                return fail(BLD_ERR_INVALID_CONFIG, "no warp y transform of radix %d", c.wfft);
            default: return fail(BLD_ERR_INVALID_CONFIG, "no warp y transform of radix %d", c.wfft);
        }
    }
    CUDA_TRY(cudaGetLastError());
    return BLD_OK;
}


template <typename R>
int setup_y() {
    BLD_TRY(upload_codelet_tables());
    BLD_SET((k_inv_y<R, 0>));
    BLD_SET((k_fwd_y<R, 0>));
    BLD_SET((k_inv_y<R, 2>));
    BLD_SET((k_fwd_y<R, 2>));
    BLD_SET((k_inv_y<R, 3>));
    BLD_SET((k_fwd_y<R, 3>));
    BLD_SET((k_inv_y<R, 4>));
    BLD_SET((k_fwd_y<R, 4>));
    BLD_SET((k_inv_y<R, 6>));
    BLD_SET((k_fwd_y<R, 6>));
    BLD_SET((k_inv_y<R, 8>));
    BLD_SET((k_fwd_y<R, 8>));
    BLD_SET((k_inv_y<R, 9>));
    BLD_SET((k_fwd_y<R, 9>));
    BLD_SET((k_inv_y<R, 12>));
    BLD_SET((k_fwd_y<R, 12>));
    BLD_SET((k_inv_y<R, 16>));
    BLD_SET((k_fwd_y<R, 16>));
    if constexpr (sizeof(R) == 4) {
        BLD_SET((k_inv_y<R, 24>));
        BLD_SET((k_fwd_y<R, 24>));
    }
    BLD_SET((k_inv_y_all<R>));
    BLD_SET((k_fwd_y_all<R>));
#define BLD_SET_Y2(P)                                                                                  \
    BLD_SET((k_inv_y2<R, y2_radix_a(P), y2_radix_b(P), y2_min_blocks_inv<R>(y2_radix_b(P) * BLD_Y2_NL)>)); \
    BLD_SET((k_fwd_y2<R, y2_radix_a(P), y2_radix_b(P), y2_min_blocks<R>(y2_radix_b(P) * BLD_Y2_NL)>)); \
    BLD_SET((k_fwd_y2<R, y2_radix_a(P), y2_radix_b(P), 3, 8, 4>));                                                                   \
    BLD_SET((k_inv_y2<R, y2_radix_a(P), y2_radix_b(P), sizeof(R) == 8 ? 3 : 4, 8>));                                                \
    if constexpr (sizeof(R) == 4)                                                                    \
        BLD_SET((k_fwd_y2<R, y2_radix_a(P), y2_radix_b(P), y2_min_blocks<R>(y2_radix_b(P) * BLD_Y2_NL), BLD_Y2_NL, 2>));
    BLD_SET_Y2(64)
    BLD_SET_Y2(96)
    BLD_SET_Y2(128)
    BLD_SET_Y2(144)
    BLD_SET_Y2(192)
    BLD_SET_Y2(256)
    BLD_SET_Y2(288)
    if constexpr (sizeof(R) == 4) {
        BLD_SET_Y2(384)
        BLD_SET_Y2(512)
        BLD_SET_Y2(768)
    }
#undef BLD_SET_Y2
#define BLD_SET_Y3(P) BLD_SET((k_inv_y3<R, y2_radix_a(P), y2_radix_b(P)>));
    BLD_SET_Y3(64)
    BLD_SET_Y3(96)
    BLD_SET_Y3(128)
    BLD_SET_Y3(144)
    BLD_SET_Y3(192)
    BLD_SET_Y3(256)
    BLD_SET_Y3(288)
    if constexpr (sizeof(R) == 4) {
        BLD_SET_Y3(384)
        BLD_SET_Y3(512)
        BLD_SET_Y3(768)
    }
#undef BLD_SET_Y3
    return BLD_OK;
}

template <typename R>
cudaError_t wait_limit_y(long long cycles) {
    return cudaMemcpyToSymbol(g_bld_wait_limit, &cycles, sizeof(cycles));
}

}  // namespace bld
