// Host interface of the line y passes (bld_ylines.cuh), which are compiled in
// translation units of their own (per direction, kind of space and precision).
#pragma once

#include <cuda_runtime.h>

#include "bld_kernels.cuh"
#include "bld_xrow.h"

namespace bld_yl {

// shape of the kernel compiled for P2 = A B: lines per block, blocks per SM the registers
// are held to; A = 0 where there is none
struct Shape {
    int A = 0, B = 0, NL = 16, MINB = 1;
};

// the radices with the smallest larger one, A a multiple of `ma`, B of `mb`
constexpr void factor(Shape& s, int P, int ma, int mb) {
    int best = 1 << 30;
    for (int b = 2; b <= 32; ++b) {
        if (P % b || !bld_row::codelet(b) || !bld_row::codelet(P / b) || (P / b) % ma || b % mb) continue;
        const int a = P / b, larger = a > b ? a : b;
        if (larger <= best) {
            best = larger;
            s.A = a;
            s.B = b;
        }
    }
}
// most blocks of `threads` per SM at `regs` registers a thread (16384 per scheduler)
constexpr int blocks(int threads, int regs) {
    int n = 1;
    while (n < 16 && ((n + 1) * ((threads + 31) / 32) + 3) / 4 * 32 * regs <= 16384 && (n + 1) * threads <= 2048) ++n;
    return n;
}

// registers a thread: the fewest that hold the larger radix with at most a little spilling
// (inverse 288 points single 56 / 72 / 80: 64 / 69 / 81 us; 192 points double 80 / 96 /
// 126: 185 / 201 / 236 us; 768 points single 64 / 80 / 128: 177 / 168 / 200 us)
constexpr int regs(int larger, bool fp32) {
    return fp32 ? (larger <= 12 ? 48 : (larger <= 16 ? 64 : (larger <= 24 ? 56 : 80)))
                : (larger <= 12 ? 64 : (larger <= 16 ? 80 : 96));
}
// Lines per block: 16, whose rows fill a wavefront (128^2 x 512 double, 8 against 16 lines:
// inverse 140 / 136, forward 131 / 122 us); 8 for the shortest transforms (more blocks on
// small grids), for radices whose 16 lines take more than 384 threads, and where they take
// more than 80 KB of shared memory.  Blocks per SM: as many as those registers and the
// shared memory allow.
constexpr Shape line_shape(int P, bool fp32, int ma, int mb, int sets) {
    Shape s;
    if (P < 12 || P > (fp32 ? 768 : 432)) return s;
    factor(s, P, ma, mb);
    if (!s.A) return s;
    const int larger = s.A > s.B ? s.A : s.B, csz = fp32 ? 8 : 16;
    s.NL = P <= 48 || larger > (fp32 ? 24 : 18) || (P + sets * 16 * P) * csz > 80 * 1024 ? 8 : 16;
    const int by_regs = blocks(larger * s.NL, regs(larger, fp32));
    const int by_smem = 227 * 1024 / ((P + sets * s.NL * (P + 32)) * csz + 1024);
    s.MINB = by_regs < by_smem ? by_regs : (by_smem > 1 ? by_smem : 1);
    return s;
}
// the pruned radix is a multiple of 3 with the 3/2 rule, the halved one even
constexpr Shape inv_shape(int P, bool fp32, bool sgs) {
    return line_shape(P, fp32, sgs ? 2 : (P % 3 == 0 ? 3 : 1), 1, 1);
}
constexpr Shape fwd_shape(int P, bool fp32, bool sgs) {
    return line_shape(P, fp32, 1, !sgs && P % 3 == 0 ? 3 : 1, sgs ? 2 : 1);
}

// the advection sizes compiled (the in-place x kernels', and 512); the Smagorinsky ones are theirs
#define BLD_YL_ADV_SIZES(X) BLD_ROW_ADV_SIZES(X) X(512)

inline bool compiled(int P, bool fp32, bool sgs) {
    if (sgs) {
#define X(N) if (P == N) return inv_shape(N, fp32, true).A > 0 && fwd_shape(N, fp32, true).A > 0;
        BLD_ROW_SGS_SIZES(X)
#undef X
    } else {
#define X(N) if (P == N) return inv_shape(N, fp32, false).A > 0 && fwd_shape(N, fp32, false).A > 0;
        BLD_YL_ADV_SIZES(X)
#undef X
    }
    return false;
}

// per translation unit: upload of the codelet twiddles to the current device, and the launch
// for args.P2 over nm members (cudaErrorInvalidValue where no kernel is compiled)
#define BLD_YL_UNITS(X) X(adv64) X(adv32) X(sgs64) X(sgs32)
#define X(U)                                                                         \
    cudaError_t init_inv_##U();                                                      \
    cudaError_t init_fwd_##U();                                                      \
    cudaError_t launch_inv_##U(const InvYArgs& a, int nm, cudaStream_t st);          \
    cudaError_t launch_fwd_##U(const FwdYArgs& a, int nm, cudaStream_t st);
BLD_YL_UNITS(X)
#undef X

}  // namespace bld_yl
