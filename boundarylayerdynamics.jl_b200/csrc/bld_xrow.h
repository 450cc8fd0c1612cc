// Host interface of the in-place x kernels (bld_xrows.cuh), which are compiled in
// translation units of their own (one per kernel and precision).
#pragma once

#include <cuda_runtime.h>

#include "bld_xargs.cuh"

namespace bld_row {

// shape of the kernel compiled for P1 = A B: rows per block, threads, blocks per SM the
// registers are held to, forward lines in their own buffer; A = 0 where there is none
struct Shape {
    int A = 0, B = 0, NR = 2, T = 96, MINB = 1;
    bool sepf = true;
};

constexpr bool codelet(int n) {
    return n == 2 || n == 3 || n == 4 || n == 5 || n == 6 || n == 7 || n == 8 || n == 9 || n == 10 || n == 12 ||
           n == 14 || n == 15 || n == 16 || n == 18 || n == 24 || n == 32;
}

// A (a multiple of 3 for advection with the 3/2 rule, even for the Smagorinsky model)
// times B with the smallest larger radix (registers); among equals the larger B in
// single and the larger A in double precision (128 points: 8 x 16 against 16 x 8,
// single 47 against 52 us, double 86 against 78 us at 128^2 x 64)
constexpr void factor(Shape& s, int P, bool fp32, int multiple) {
    int best = 1 << 30;
    for (int b = 2; b <= 32; ++b) {
        if (P % b || !codelet(b) || !codelet(P / b) || (P / b) % multiple) continue;
        const int a = P / b, larger = a > b ? a : b;
        if (larger < best || (larger == best && fp32)) {
            best = larger;
            s.A = a;
            s.B = b;
        }
    }
}

// Advection.  Threads: about one per task of the inverse passes, so that few idle in the
// others (288 points, double: 96 / 128 / 192 threads 0.195 / 0.181 / 0.237 ms at
// 192^2 x 96, single 0.099 / 0.105 / 0.114 ms).  Four rows per block up to 216 points in
// single precision (two against four rows: 96 points 103 / 89 us at 64^2 x 768, 144 points
// 136 / 117 us at 96^2 x 512), two elsewhere (registers, shared memory).  Blocks per SM:
// the most whose register cap does not spill.  384 points and above in double precision
// share the line buffer between both directions, for three blocks per SM (0.234 against
// 0.244 ms with two at 256^2 x 64).
constexpr Shape adv_shape(int P, bool fp32) {
    Shape s;
    if (P < 12 || P > (fp32 ? 768 : 432) || P == 512) return s;   // 512: no faster than k_adv_x2
    factor(s, P, fp32, P % 3 == 0 ? 3 : 1);
    if (P == 144) s.A = 9, s.B = 16;
    if (P == 288) s.A = 18, s.B = 16;
    if (P == 384) s.A = 24, s.B = 16;
    if (!s.A) return s;
    const int larger = s.A > s.B ? s.A : s.B;
    if (P <= 48) {
        s.T = 64;
        s.MINB = fp32 ? 8 : 6;
    } else if (fp32 && P <= 216) {
        s.NR = 4;
        s.T = P <= 108 ? 96 : (P <= 162 ? 128 : 192);
        s.MINB = s.T == 96 ? 7 : (s.T == 128 ? 5 : 4);
    } else if (fp32) {
        s.T = larger > 24 ? 192 : 96;
        s.MINB = larger > 24 ? 2 : (larger >= 18 ? 5 : 6);
    } else {
        s.T = P > 216 && P < 384 ? 128 : 96;
        s.MINB = s.T == 128 || P >= 384 ? 3 : (larger <= 9 || P <= 144 ? 5 : 4);
        s.sepf = P < 384;
    }
    return s;
}

// Smagorinsky (P1 = 2 k1max + 2).  Single precision: two rows per block, one above 288
// points, and one thread per task of the last forward pass (four lines a row of B tasks:
// 64 points 64 / 96 / 128 threads 111 / 138 / 130 us at 64^2 x 768; 256 points, one row and
// 64 threads 280, two rows and 128 threads 240 us at 256^2 x 128).  Double precision, whose
// carried values take 26 registers a point: one row above 144 points.
constexpr Shape sgs_shape(int P, bool fp32) {
    Shape s;
    if (P < 12 || P > (fp32 ? 512 : 324)) return s;
    factor(s, P, fp32, 2);
    if (P == 96 && fp32) s.A = 6, s.B = 16;
    if (!s.A) return s;
    const int larger = s.A > s.B ? s.A : s.B;
    if (fp32) {
        s.NR = P <= 288 || P % 4 ? 2 : 1;
        s.T = (4 * s.NR * s.B + 31) / 32 * 32;
        if (s.T > 160) s.T = 160;
        s.MINB = s.T == 32 ? 16 : (s.T == 64 ? 8 : (s.T == 96 ? 5 : (s.T == 160 || s.NR == 1 ? 3 : (P == 128 ? 5 : 4))));
    } else {
        s.NR = P <= 144 ? 2 : 1;
        s.T = P <= 72 ? 64 : 96;
        s.MINB = s.T == 96 ? 4 : (larger <= 8 ? 8 : 6);
    }
    return s;
}

// the P1 compiled (adv_shape / sgs_shape decide per precision)
#define BLD_ROW_ADV_SIZES(X) \
    X(12) X(16) X(18) X(24) X(32) X(36) X(48) X(54) X(64) X(72) X(96) X(108) X(128) X(144) X(162) X(192) X(216) \
    X(256) X(288) X(324) X(384) X(432) X(576) X(768)
#define BLD_ROW_SGS_SIZES(X) \
    X(12) X(14) X(16) X(18) X(20) X(24) X(28) X(30) X(32) X(36) X(40) X(42) X(48) X(50) X(54) X(56) X(60) X(64) \
    X(70) X(72) X(80) X(84) X(90) X(96) X(98) X(100) X(108) X(112) X(120) X(126) X(128) X(140) X(144) X(150) \
    X(160) X(162) X(168) X(180) X(192) X(196) X(210) X(216) X(224) X(240) X(252) X(256) X(270) X(288) X(320) \
    X(324) X(336) X(360) X(384) X(432) X(448) X(480) X(512)

inline bool adv_compiled(int P, bool fp32) {
#define X(N) if (P == N) return adv_shape(N, fp32).A > 0;
    BLD_ROW_ADV_SIZES(X)
#undef X
    return false;
}
inline bool sgs_compiled(int P, bool fp32) {
#define X(N) if (P == N) return sgs_shape(N, fp32).A > 0;
    BLD_ROW_SGS_SIZES(X)
#undef X
    return false;
}

// copy the codelet twiddles (h_wtab64 / h_wtab32) to the current device
cudaError_t init_adv64();
cudaError_t init_adv32();
cudaError_t init_sgs64();
cudaError_t init_sgs32();

// enqueue the kernel for a.P1 over nm members and `nchunks` z chunks of a.zchunk layers;
// cudaErrorInvalidValue where none is compiled
cudaError_t launch_adv64(const XArgs& a, int nchunks, int nm, cudaStream_t st);
cudaError_t launch_adv32(const XArgs& a, int nchunks, int nm, cudaStream_t st);
cudaError_t launch_sgs64(const XArgs& a, int nchunks, int nm, cudaStream_t st);
cudaError_t launch_sgs32(const XArgs& a, int nchunks, int nm, cudaStream_t st);

}  // namespace bld_row
