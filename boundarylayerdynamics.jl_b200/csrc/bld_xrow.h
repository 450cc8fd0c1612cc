// Host interface of the in-place x kernels (bld_xrows.cuh), which are compiled in
// translation units of their own (one per kernel and precision).
#pragma once

#include <cuda_runtime.h>

#include "bld_xargs.cuh"

namespace bld_row {

// shape of the kernel compiled for P1 = A B: rows per block, threads, blocks per SM the
// registers are held to, advection's forward lines in their own buffer; A = 0 where there is none
struct Shape {
    int A = 0, B = 0, NR = 2, T = 96, MINB = 1;
    bool sepf = true;
};

constexpr bool codelet(int n) {
    return n == 2 || n == 3 || n == 4 || n == 5 || n == 6 || n == 7 || n == 8 || n == 9 || n == 10 || n == 12 ||
           n == 14 || n == 15 || n == 16 || n == 18 || n == 24 || n == 32;
}

// A (a multiple of 3 for advection with the 3/2 rule, even for the Smagorinsky model)
// times B with the smallest larger radix (registers).  Among equals: the larger B in
// single precision, and in double precision for advection where it fills the lanes of
// the last forward pass (128 points, double, 8 x 16 against 16 x 8: advection 211 / 228 us
// at 84^2 x 512), else the larger A (Smagorinsky 86 / 78 us at 128^2 x 64).  A warp has
// 32 / B lines in that pass; where that B leaves lanes idle, B = 16 takes its place if the
// larger radix grows by no more than a third (us, before against now: advection 144
// points single 164 / 117, double 255 / 227 at 96^2 x 512; Smagorinsky single 96 points
// 197 / 170, 288 238 / 204, 384 284 / 263), but not for the Smagorinsky model in double
// precision, where the larger first radix holds its own (192 points, 16 x 12 against
// 12 x 16, 192^2 x 32 116 / 121 us).
constexpr void factor(Shape& s, int P, bool fp32, bool adv, int multiple) {
    int best = 1 << 30;
    for (int b = 2; b <= 32; ++b) {
        if (P % b || !codelet(b) || !codelet(P / b) || (P / b) % multiple) continue;
        const int a = P / b, larger = a > b ? a : b;
        if (larger < best || (larger == best && (fp32 || (adv && 32 % b == 0)))) {
            best = larger;
            s.A = a;
            s.B = b;
        }
    }
    if (!s.A || 32 % s.B == 0 || P % 16 || !(adv || fp32)) return;
    const int a = P / 16, larger = a > 16 ? a : 16;
    if (codelet(a) && a % multiple == 0 && 3 * larger <= 4 * best) {
        s.A = a;
        s.B = 16;
    }
}

// Advection.  Threads: about one per task of the inverse passes, so that few idle in the
// others (288 points, double: 96 / 128 / 192 threads 0.195 / 0.181 / 0.237 ms at
// 192^2 x 96, single 0.099 / 0.105 / 0.114 ms).  Four rows per block up to 216 points in
// single precision (two against four rows: 96 points 103 / 89 us at 64^2 x 768, 144 points
// 136 / 117 us at 96^2 x 512), two elsewhere (registers, shared memory) but for radices up
// to 8 in double precision where no third of the spectrum is empty: there every task has
// all its inputs, and two rows leave half of the threads without one (64 points 100 / 72 us
// at 42^2 x 768, k_adv_x2 84; with the empty third four rows are slower on a grid that does
// not fill the chip: 96 points 14.6 / 16.7 us at 64^2 x 32).  Blocks per SM: the most whose
// register cap does not spill (256 points, single, six / five blocks: 123 / 115 us at
// 168^2 x 128).  384 points and above in double precision share the line buffer between
// both directions, for three blocks per SM (0.234 against 0.244 ms with two at 256^2 x 64).
constexpr Shape adv_shape(int P, bool fp32) {
    Shape s;
    if (P < 12 || P > (fp32 ? 768 : 432) || P == 512) return s;   // 512: no faster than k_adv_x2
    factor(s, P, fp32, true, P % 3 == 0 ? 3 : 1);
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
        s.MINB = larger > 24 ? 2 : 5;
    } else {
        s.NR = P % 3 && larger <= 8 ? 4 : 2;
        s.T = P > 216 && P < 384 ? 128 : 96;
        s.MINB = s.T == 128 || P >= 384 ? 3 : (larger <= 9 || P <= 144 ? 5 : 4);
        s.sepf = P < 384;
    }
    return s;
}

// Smagorinsky (P1 = 2 k1max + 2).  Single precision: two rows per block, one above 288
// points, and one thread per task of the last forward pass (four lines a row of B tasks:
// 64 points 64 / 96 / 128 threads 111 / 138 / 130 us at 64^2 x 768; 256 points, one row and
// 64 threads 280, two rows and 128 threads 240 us at 256^2 x 128), but with one row at least
// 96 for the wide first radices (360 points, 24 x 15: 64 / 96 threads 318 / 278 us at
// 360^2 x 48).  Blocks per SM of 128 threads as the registers of the first radix allow
// where every lane works and the lines are long enough to fill them (8 x 16, 128^2 x 256,
// five / four blocks 148 / 158 us, 10 x 16 225 / 214, 18 x 16 four / three 221 / 204; but
// 6 x 16, 96^2 x 48, five / four 31 / 29, eight of them 150 / 139), four where some lanes idle
// (8 x 14, ten 112^2 x 16, five / four 93 / 84, 18 x 15, two 270^2 x 16, four / three
// 98 / 128); with one row the most that do not spill
// (five / four / three blocks at 324 points 305 / 286 / 285 us, 384 321 / 262 / 263, 432
// 529 / 401 / 412, 480 490 / 407 / 358).
// Double precision, whose carried values take 26 registers a point: one row above 144
// points.
constexpr Shape sgs_shape(int P, bool fp32) {
    Shape s;
    if (P < 12 || P > (fp32 ? 512 : 324)) return s;
    factor(s, P, fp32, false, 2);
    if (!s.A) return s;
    const int larger = s.A > s.B ? s.A : s.B;
    if (fp32) {
        s.NR = P <= 288 || P % 4 ? 2 : 1;
        s.T = (4 * s.NR * s.B + 31) / 32 * 32;
        if (s.T > 160) s.T = 160;
        if (s.NR == 1 && s.T < 96) s.T = 96;
        s.MINB = s.T == 32 ? 16 : (s.T == 64 ? 8 : (s.T == 96 ? 5 : 3));
        if (s.T == 128) s.MINB = 32 % s.B || P < 128 ? 4 : (s.A <= 8 ? 5 : (s.A <= 16 ? 4 : 3));
        if (s.NR == 1) s.MINB = larger <= 24 ? 4 : 3;
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
