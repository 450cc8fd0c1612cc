// The handle, the physical-domain spaces and the host helpers shared by the engine's
// translation units: the C ABI with the schedules (bld_capi.cu) and the kernel
// families that are compiled on their own (bld_family_*.cu, bld_xrow_*.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstdint>
#include <cstring>
#include <initializer_list>
#include <map>
#include <string>
#include <utility>
#include <vector>

#include "bld.h"
#include "bld_kernels.cuh"
#include "bld_warpx.cuh"
#include "bld_advx2.cuh"
#include "bld_sgsx2.cuh"
#include "bld_xrow.h"

namespace bld {

// sets the calling thread's error message and returns `code`
int fail(int code, const char* fmt, ...);

#define CUDA_TRY(expr)                                                                      \
    do {                                                                                    \
        cudaError_t e_ = (expr);                                                            \
        if (e_ != cudaSuccess)                                                              \
            return fail(e_ == cudaErrorMemoryAllocation ? BLD_ERR_OUT_OF_MEMORY : BLD_ERR_CUDA, \
                        "%s: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__);  \
    } while (0)

#define BLD_TRY(expr)          \
    do {                       \
        int s_ = (expr);       \
        if (s_ != BLD_OK) return s_; \
    } while (0)

// ---------------------------------------------------------------- FFT sizes and plans
inline bool smooth_of(int n, std::initializer_list<int> primes) {
    if (n < 2) return false;
    for (int p : primes)
        while (n % p == 0) n /= p;
    return n == 1;
}
inline bool smooth23(int n) { return smooth_of(n, {2, 3}); }
// sizes the block Stockham kernels transform: products of 2, 3, 5 and 7
inline bool smooth2357(int n) { return smooth_of(n, {2, 3, 5, 7}); }

inline int next_even_smooth(int n) {
    int m = std::max(n, 2);
    while (!(m % 2 == 0 && smooth23(m))) ++m;
    return m;
}

// Fewest Stockham stages whose radices are register codelet sizes, then the
// smallest largest radix (register pressure), capped at BLD_FP32_MAXR / BLD_FP64_MAXR;
// nst = 0 if no such plan of at most four stages exists.
inline FftPlan make_plan(int n, bool fp32 = false) {
    static const int rads[] = {32, 24, 18, 16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    const int cap = fp32 ? BLD_FP32_MAXR : BLD_FP64_MAXR;
    FftPlan best{};
    best.n = n;
    best.nst = 0;
    int best_st = 99, best_max = 99;
    int seq[6];
    // depth-first search over radix sequences (n <= 1024 of 2, 3, 5, 7 needs at most 4 stages of <= 18)
    auto dfs = [&](auto&& self, int rem, int depth, int mx) -> void {
        if (depth > 4 || depth > best_st) return;
        if (rem == 1) {
            if (depth < best_st || (depth == best_st && mx < best_max)) {
                best_st = depth;
                best_max = mx;
                best.nst = depth;
                for (int i = 0; i < depth; ++i) best.radix[i] = seq[i];
            }
            return;
        }
        for (int r : rads) {
            if (r > cap || rem % r) continue;
            seq[depth] = r;
            self(self, rem / r, depth + 1, std::max(mx, r));
        }
    };
    dfs(dfs, n, 0, 0);
    return best;
}

// quadratic-dealiasing size of the reference (src/physical_space.jl:49-56)
inline int pdsize_quadratic(int kmax) {
    const double l = std::log2(1.0 + kmax);
    if (l == std::floor(l)) return 3 * kmax + 3;
    return 3 * kmax + ((kmax % 2 == 1) ? 1 : 2);
}

struct DevTw {
    void* d64 = nullptr;
    void* d32 = nullptr;
};

// a y-pass variant: per-term (per-field) blocks with a two-buffer FFT, or one
// block for all terms (fields) of a layer with an in-place FFT
struct YCfg {
    int all = 0;
    int NL = 4;    // k1 lines per term (per field and line set)
    int thr = 256;
    int wfft = 0;  // per-term kernels: radix of the warp transform (P2 = 32 wfft), 0 = block stages
    int tp = 0;    // 1: two-pass kernels (k_inv_y2 / k_fwd_y2), BLD_Y2_NL lines, P2 = A * B;
                   // 2: inverse pass with TMA-staged tiles (k_inv_y3), BLD_Y3_NL lines;
                   // 3: two-pass kernels on 8 lines (forward: 3 blocks per SM, 4 outputs in flight;
                   //    inverse: 3 blocks per SM in double, 4 in single precision);
                   // 4: forward two-pass kernel, single precision, 2 outputs in flight
    int zc = 1;    // tp 2: layer chunks (blocks along z)
};

// radices of the warp y transforms compiled for the per-term y kernels
// (24 in single precision only)
inline bool wfft_radix_ok(int r, bool fp32) {
    return r == 2 || r == 3 || r == 4 || r == 6 || r == 8 || r == 9 || r == 12 || r == 16 || (fp32 && r == 24);
}

struct Space {
    bool on = false;
    int P1 = 0, P2 = 0, ref_P1 = 0, ref_P2 = 0;
    FftPlan plan1{}, plan2{};
    int ntin = 0, ntout = 0;
    void* min = nullptr;
    void* mout = nullptr;
    long long min_ms = 0, mout_ms = 0;  // elements per member
    int YT = 1, PPT = 1, zchunk = 1, nchunks = 1;  // x kernels: rows per block, points per thread, z chunks
    int xw = 0;                                     // > 0: warp-per-row x kernel with xw warps per block
    int xwmb = 1;                                   // warp-per-row kernel: register cap (min blocks of 128 threads)
    int zmult = 2;                                  // x kernels: z-chunk count multiplier in halves (autotuned)
    int xb = 0;                                     // block of warps per row (advection): 1 three warps, 2 five (pipelined)
    int x2 = 0;                                     // 1 + V: two-pass shared-memory x kernel k_adv_x2<.., V> (advection)
    int sx2 = 0;                                    // SGS block x kernel with two-pass line transforms: 1 plain,
                                                    // 2 registers capped for two blocks of 256 threads per SM,
                                                    // 3 / 4 as 1 / 2 with the input rows staged by bulk copies
    int sxk = 0;                                    // 1 + V: SGS x kernel k_sgs_x2<.., V> (rows staged by bulk copies, two-pass lines)
    int xrow = 0;                                   // 1: in-place x kernel k_adv_row / bld_row::k_sgs_x (bld_xrows.cuh); the SGS
                                                    // space then has six mixed terms each way instead of nine and eight
    int xr = 0;                                     // block x kernels: warp-transform radix (P1 = 32 xr), 0 = Stockham
    int fsets = 1;                                  // forward line sets (2 when a D2 contribution exists)
    YCfg inv, fwd;                                  // y-pass variants (chosen by the autotuner)
    int yl = 0;                                     // 1: the line y passes k_inv_yl / k_fwd_yl (bld_ylines.cuh) instead
};

}  // namespace bld

using namespace bld;

struct bld_handle {
    bld_config cfg{};
    int device = 0;
    int B = 1;
    Geo g{};
    bool fp32 = false;
    cudaStream_t stream = nullptr;
    // state and integrator buffers [member][vel1|vel2|vel3]
    double2* u = nullptr;
    double2* t = nullptr;
    double2* du = nullptr;
    double2* dp = nullptr;
    double2* io = nullptr;     // staging for host-buffer calls
    double2* io2 = nullptr;
    double2* pscr = nullptr;
    double* gamma = nullptr;
    // tables
    double *d1 = nullptr, *d2 = nullptr, *DD1 = nullptr, *DD2 = nullptr;
    double *alpha_c = nullptr, *alpha_i = nullptr, *alpha_ext = nullptr, *mean_w = nullptr;
    double* inv_alpha_c = nullptr;   // 1 / alpha_c (the projections' divergence)
    double *lc2 = nullptr, *li2 = nullptr, *wall = nullptr, *src = nullptr, *mean_val = nullptr;
    long long* wait_limit = nullptr;   // device address of the limit of bounded waits
    int* flag = nullptr;
    int* flag_host = nullptr;
    std::vector<int> diverged;   // members whose rates turned non-finite since the last bld_get_diverged
    int* active = nullptr;        // [members] device mask of active ensemble slots
    std::vector<int> active_host;
    bool mask_on = false;        // the active mask applies to whole-ensemble steps only
    int proj_variant = 1;        // 0: column kernel, 1/2: z-segmented kernel, 3: with a shared tile (autotuned)
    int proj_tile = 0;           // LN > 0: projections of stored stage values by k_project_tile<.., LN> (autotuned)
    int proj_pipe = 0;           // 1: ... by its persistent two-stage form k_project_pipe<.., LN> (autotuned)
    double* prof_acc = nullptr;  // [members][3][n3+1] time integral of the mean profiles
    double* prof_prev = nullptr; // [members][3][n3+1] last sample
    bool prof_on = false;        // step graphs sample the profiles after every step
    std::vector<double> tab_dx3c, tab_dx3i, tab_x3c, tab_x3i;  // copies of the mapping tables
    std::vector<double> member_cs, member_z0;                  // current per-member SGS parameters
    std::map<int, DevTw> tw;
    Space adv, sgs;
    // physical-domain transforms at the default size
    int Pd1 = 0, Pd2 = 0;
    void* pd_buf = nullptr;     // double [nz][Pd2][Pd1]
    void* pd_mixed = nullptr;   // double2 [nz][Pd2][K1]
    // progress statistics (allocated by the first bld_progress_stats call)
    double* prog_small = nullptr;  // per-layer sums and maxima
    void* prog_buf = nullptr;      // double [n3][P2][P1] at the largest physical size
    void* prog_mixed = nullptr;    // double2 [n3][P2][K1]
    // host-side copies used by launches
    double w_lo = 0, w_hi = 0;
    int dyn_lo = 0, dyn_hi = 0;
    double d3_scale = 1.0;                                        // XArgs::d3_scale and its tables
    double *d3_alpha_c = nullptr, *d3_alpha_i = nullptr;
    Linear lin{};
    bool slope_valid = false;
    bool ab2_started = false;
    double ab2_dt = 0;
    std::map<std::pair<int, double>, cudaGraphExec_t> graphs;
    std::map<std::pair<int, double>, cudaGraph_t> graph_src;   // kept for ensemble parent graphs
    std::map<std::pair<int, double>, int64_t> enqueued_steps;  // steps that ran without a graph, per method and dt
    std::map<std::vector<const void*>, cudaGraphExec_t> ens_graphs;  // parent graphs led by this handle
    size_t bytes = 0;
    int proj_euler = 0;          // 1: the Euler stage of a step by k_project_tile too (autotuned)
    // kernels enqueued now may be set up while the one before them on the stream ends
    // (overlapped launches; off for the first kernel of a schedule and after a join)
    bool overlap = false;
    cudaStream_t side = nullptr;   // second branch of the right-hand side (with both physical spaces)
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
};

namespace bld {

inline int dalloc(bld_handle* h, void** p, size_t bytes) {
    if (bytes == 0) bytes = 16;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) return fail(BLD_ERR_OUT_OF_MEMORY, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
    h->bytes += bytes;
    return BLD_OK;
}

template <typename T>
int upload(bld_handle* h, T** dst, const std::vector<T>& v) {
    BLD_TRY(dalloc(h, (void**)dst, v.size() * sizeof(T)));
    if (!v.empty()) CUDA_TRY(cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return BLD_OK;
}

inline int twiddles(bld_handle* h, int n) {
    if (h->tw.count(n)) return BLD_OK;
    std::vector<double2> w64(n);
    std::vector<float2> w32(n);
    for (int m = 0; m < n; ++m) {
        const long double ang = -2.0L * 3.14159265358979323846264338327950288L * (long double)m / (long double)n;
        const long double c = cosl(ang), s = sinl(ang);
        w64[m] = make_double2((double)c, (double)s);
        w32[m] = make_float2((float)c, (float)s);
    }
    DevTw t;
    BLD_TRY(dalloc(h, &t.d64, n * sizeof(double2)));
    BLD_TRY(dalloc(h, &t.d32, n * sizeof(float2)));
    CUDA_TRY(cudaMemcpy(t.d64, w64.data(), n * sizeof(double2), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(t.d32, w32.data(), n * sizeof(float2), cudaMemcpyHostToDevice));
    h->tw[n] = t;
    return BLD_OK;
}

inline const void* twp(const bld_handle* h, int n, bool fp32) {
    const DevTw& t = h->tw.at(n);
    return fp32 ? t.d32 : t.d64;
}

inline size_t csize(bool fp32) { return fp32 ? sizeof(float2) : sizeof(double2); }

// y-pass lines per block: shared memory <= ~100 KB and outputs per thread <= 16
// y-pass lines per block: the largest of 16 (single) / 8, 4, 2 whose two
// shared line buffers (times `sets`) and twiddles stay within ~110 KB
inline int pick_y(int P2, bool fp32, int sets) {
    const size_t cs = csize(fp32);
    int NL = fp32 ? 16 : 8;
    while (NL > 2 && (size_t)(P2 + 2 * P2 * sets * NL) * cs > 110 * 1024) NL /= 2;
    return NL;
}

// shape of the in-place x kernel of a space
inline bld_row::Shape row_shape(const bld_handle* h, const Space& s) {
    return &s == &h->sgs ? bld_row::sgs_shape(s.P1, h->fp32) : bld_row::adv_shape(s.P1, h->fp32);
}

// choose tiles for a physical-domain space
// z chunks of the x kernels for the current rows per block: enough blocks to
// fill the GPU a few times over, at least 8 layers per chunk
inline void x_chunks(const bld_handle* h, Space& s) {
    const int n3 = h->g.n3;
    const int rows = s.xrow ? row_shape(h, s).NR : s.x2 ? x2_rows((int)csize(h->fp32), s.P1, s.x2 - 1)
                           : (s.sxk ? sx2_rows((int)csize(h->fp32), s.P1, s.sxk - 1) : (s.xb ? 1 : (s.xw ? s.xw : s.YT)));
    const long long blocks_per_chunk = (long long)((s.P2 + rows - 1) / rows) * h->B;
    int want = (int)std::max<long long>(1, (900 + blocks_per_chunk - 1) / blocks_per_chunk);
    want = std::min(want, std::max(1, n3 / 8));
    // the autotuner may ask for more chunks (shorter streams, more blocks: a
    // smaller partial last wave), down to 4 layers per chunk
    // (the row kernels, with their short layers, down to one)
    want = std::min(std::max(1, want * s.zmult / 2), std::max(1, s.xrow ? n3 : n3 / 4));
    s.zchunk = (n3 + want - 1) / want;
    s.nchunks = (n3 + s.zchunk - 1) / s.zchunk;
}

// (rows per block, points per thread) candidates of the x kernels: blocks of
// 32..256 threads whose two line buffers fit in 150 KB of shared memory
inline std::vector<std::pair<int, int>> x_candidates(const bld_handle* h, const Space& s, bool is_adv) {
    std::vector<std::pair<int, int>> out;
    const int lines = is_adv ? 3 : 5;
    for (int yt : {1, 2, 4}) {
        if (s.P2 % yt || yt * s.P1 > 1024) continue;
        if ((size_t)(s.P1 + 2 * lines * yt * s.P1) * csize(h->fp32) > 150 * 1024) continue;
        for (int ppt = 1; ppt <= 4; ++ppt) {
            const int pts = yt * s.P1;
            if (pts % ppt) continue;
            const int thr = pts / ppt;
            if (thr > 256 || thr < 32) continue;
            out.emplace_back(yt, ppt);
        }
    }
    return out;
}

inline void tile_space(const bld_handle* h, Space& s, bool is_adv) {
    // initial choice near 96 (advection, double) / 128 (SGS, double) / 192 (single)
    // threads; the autotuner replaces it with the measured best
    const int target = h->fp32 ? 192 : (is_adv ? 96 : 128);
    int best = 1 << 30;
    s.YT = 1;
    s.PPT = 0;
    for (auto c : x_candidates(h, s, is_adv)) {
        const int thr = c.first * s.P1 / c.second;
        const int score = std::abs(thr - target) + 24 * (c.second - 1) + 8 * (c.first - 1);
        if (score < best) {
            best = score;
            s.YT = c.first;
            s.PPT = c.second;
        }
    }
    x_chunks(h, s);
}

inline size_t smem_y(int P2, int NL, bool fp32) { return (size_t)(P2 + 2 * P2 * NL) * csize(fp32); }
// per-term y kernels with `lines` lines: twiddles and two line buffers for the
// block-wide stages, or twiddles and one buffer of P2 + 32 (swizzled) positions
// on a line stride of lines + 1 for the warp transforms
inline size_t smem_y_term(int P2, int lines, int wfft, bool fp32) {
    return (size_t)(wfft ? P2 + (P2 + 32) * (lines + 1) : P2 + 2 * P2 * lines) * csize(fp32);
}
// block x kernels: twiddles and two buffers of (3 or 5) YT lines, on a line stride
// P1 + 32 (swizzled positions) with warp line transforms (xr > 0)
inline size_t smem_adv(const Space& s, bool fp32) {
    return (size_t)(s.P1 + 2 * 3 * s.YT * (s.P1 + (s.xr ? 32 : 0))) * csize(fp32);
}
// the two-pass SGS kernel stages its input rows by bulk copies when a block's
// YT rows of K1 values fill whole 16-byte units
inline bool sgs_stage_fits(const Space& s, bool fp32, int K1) { return !fp32 || K1 % 2 == 0 || s.YT % 2 == 0; }
inline bool sgs_staged(const Space& s, bool fp32, int K1) { return s.sx2 >= 3 && sgs_stage_fits(s, fp32, K1); }

inline size_t smem_sgs(const Space& s, bool fp32, int K1) {
    if (s.sx2) {
        const int A = y2_radix_a(s.P1), B = y2_radix_b(s.P1);
        const int lp = fp32 ? twopass_line<float2>(A, B) : twopass_line<double2>(A, B);
        if (sgs_staged(s, fp32, K1))
            return (size_t)sgs_stage_offset(s.P1, 5 * s.YT, lp, (int)csize(fp32)) + 128 +
                   (size_t)2 * 9 * s.YT * K1 * csize(fp32);
        return (size_t)(s.P1 + 2 * 5 * s.YT * lp) * csize(fp32);
    }
    return (size_t)(s.P1 + 2 * 5 * s.YT * (s.P1 + (s.xr ? 32 : 0))) * csize(fp32);
}

// ------------------------------------------------------------------ kernel dispatch
// threads for an in-place transform of `lines` lines (one task per thread for
// radix >= 8, up to four for smaller radices); 0 if more than 384 are needed
inline int inplace_threads(const FftPlan& pl, int lines) {
    int thr = 32;
    for (int i = 0; i < pl.nst; ++i) {
        const int r = pl.radix[i];
        const int tpt = r <= 4 ? 4 : (r == 6 ? 3 : 1);  // inplace_tpt
        const int tasks = lines * pl.n / r;
        thr = std::max(thr, (tasks + tpt - 1) / tpt);
    }
    thr = (thr + 31) / 32 * 32;
    return thr <= 384 ? thr : 0;
}

// threads of a y-pass block: enough for the widest FFT stage of `lines` lines
inline int y_threads(const FftPlan& pl, int lines) {
    int rmin = 64;
    for (int i = 0; i < pl.nst; ++i) rmin = std::min(rmin, pl.radix[i]);
    const int tasks = lines * pl.n / rmin;
    return std::min(256, std::max(64, (tasks + 31) / 32 * 32));
}

// two-pass y kernels: compiled for P2 with a factorisation y2_radix_a/b (single
// precision up to 768, double up to 288) and their registers per block count
inline bool y2_ok(int P2, bool fp32) { return y2_radix_a(P2) > 0 && (fp32 || P2 <= 288); }
inline size_t smem_y2(int P2, int lines, bool fp32) { return (size_t)P2 * (1 + lines) * csize(fp32); }

// cuTensorMapEncodeTiled from the driver, found through the runtime (the
// library links only the static CUDA runtime)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// the members' states from `base` as a float64 tensor (2 K1, K2, 3 n3 - 1, members)
// with the box (2 NL, K2, 1, 1) of k_inv_y3
inline int state_tmap(const bld_handle* h, const void* base, int nl, CUtensorMap* out) {
    const Geo& g = h->g;
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return fail(BLD_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[4] = {(cuuint64_t)(2 * g.K1), (cuuint64_t)g.K2, (cuuint64_t)(3 * g.n3 - 1), (cuuint64_t)h->B};
    const cuuint64_t strides[3] = {(cuuint64_t)g.K1 * 16, (cuuint64_t)g.F * 16, (cuuint64_t)g.mstride * 16};
    const cuuint32_t box[4] = {(cuuint32_t)(2 * nl), (cuuint32_t)g.K2, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BLD_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return BLD_OK;
}

// k_inv_y3 applies: a two-pass factorisation, whole K2 columns in one TMA box
// (K2 <= 256) and the staged tiles within the shared memory of a block
inline bool y3_ok(const bld_handle* h, int P2) {
    return y2_ok(P2, h->fp32) && h->g.K2 <= 256 &&
           y3_smem(P2, h->g.K2, (int)csize(h->fp32)) <= 227 * 1024 && encode_tiled() != nullptr;
}

// two-pass advection x kernel: compiled for P1 with a two-pass factorisation
// (single precision up to 768, double up to 288), whole row pairs per block;
// variants V = 2 (wide) in double precision, V = 3 (two rows) in single precision up to 384
inline bool x2_ok(const bld_handle* h, const Space& s, int V = 0) {
    const int cs = (int)csize(h->fp32);
    return y2_ok(s.P1, h->fp32) && s.P2 % x2_rows(cs, s.P1, V) == 0 &&
           (V == 0 || (V == 2 && !h->fp32) || (V == 3 && h->fp32 && s.P1 <= 384)) &&
           x2_smem(y2_radix_a(s.P1), y2_radix_b(s.P1), h->g.K1, cs, V) <= 227 * 1024;
}

// radices of the warp line transforms compiled into the block x kernels, and the
// points per thread that go with each (so that YT * 32 RAD / PPT threads are whole warps)
inline bool xr_radix_ok(int r) { return r == 2 || r == 3 || r == 4 || r == 6 || r == 8 || r == 9 || r == 12 || r == 16 || r == 24; }
constexpr int xr_ppt(int r) { return r <= 4 ? 1 : r <= 8 ? 2 : r <= 12 ? 3 : 4; }

// radix of the warp-per-row x kernel for P1 = 32 * radix, or 0 if no variant is compiled
template <typename R>
int warpx_radix(int P1) {
    if (P1 % 32) return 0;
    const int r = P1 / 32;
    if (sizeof(R) == 8) return (r == 2 || r == 3 || r == 4 || r == 6) ? r : 0;
    return (r == 2 || r == 3 || r == 4 || r == 6 || r == 8 || r == 9 || r == 12) ? r : 0;
}

// register caps compiled for the warp-per-row x kernel (single precision, radix >= 8)
template <typename R>
bool warpx_minb_ok(int r, int mb) {
    if (mb == 1) return true;
    return sizeof(R) == 4 && (r == 8 || r == 9 || r == 12) && (mb == 3 || mb == 4);
}

// radix of the block-of-warps x kernels for P1 = 32 * radix (16 and 24 in single
// precision only: one line of 24 FP64 complex values per lane would spill), or 0
inline int xb_radix(int P1, bool fp32) {
    if (P1 % 32) return 0;
    const int r = P1 / 32;
    if (fp32 && (r == 16 || r == 24)) return r;
    return (r == 2 || r == 3 || r == 4 || r == 6 || r == 8 || r == 9 || r == 12) ? r : 0;
}

// the register-capped two-pass SGS x kernels: single precision, P1 >= 256
// (where the uncapped kernel needs ~170 registers, one block per SM)
__host__ __device__ constexpr bool sx2_capped_size(int P) { return P >= 256; }

// SGS x kernel with two-pass line transforms: compiled for the two-pass sizes and
// one or two points per thread of the products; v = 2: the register-capped form
inline bool sx2_ok(const bld_handle* h, const Space& s, int v = 1) {
    return y2_ok(s.P1, h->fp32) && (v % 2 == 1 || (h->fp32 && sx2_capped_size(s.P1)));
}

// k_sgs_x2: compiled for the two-pass sizes; whole row groups per block
// V = 1 (two rows per block) in single precision up to P1 = 384
inline bool sxk_ok(const bld_handle* h, const Space& s, int V = 0) {
    const int cs = (int)csize(h->fp32);
    return y2_ok(s.P1, h->fp32) && (V == 0 || (h->fp32 && s.P1 <= 384)) && s.P2 % sx2_rows(cs, s.P1, V) == 0 &&
           sx2_smem(y2_radix_a(s.P1), y2_radix_b(s.P1), h->g.K1, cs, V) <= 227 * 1024;
}


// ---- kernel families compiled in their own translation units (R = double, float)
// launches of the y passes and of the x passes other than the in-place ones
template <typename R>
int launch_inv_y(bld_handle* h, const Space& s, InvYArgs a, int nm);
template <typename R>
int launch_fwd_y(bld_handle* h, const Space& s, FwdYArgs a, int nm);
template <typename R>
int launch_adv_family(bld_handle* h, const Space& s, const XArgs& a, int nm);
template <typename R>
int launch_sgs_x(bld_handle* h, const Space& s, const XArgs& a, int nm);
// once per device: the unit's codelet twiddles and its kernels' shared-memory limits
template <typename R>
int setup_y();
template <typename R>
int setup_adv();
template <typename R>
int setup_sgs();
// the unit's copy of the limit of bounded waits
template <typename R>
cudaError_t wait_limit_y(long long cycles);
template <typename R>
cudaError_t wait_limit_adv(long long cycles);
template <typename R>
cudaError_t wait_limit_sgs(long long cycles);

inline int upload_codelet_tables() {
    CUDA_TRY(cudaMemcpyToSymbol(c_wtab64, h_wtab64, sizeof(h_wtab64)));
    CUDA_TRY(cudaMemcpyToSymbol(c_wtab32, h_wtab32, sizeof(h_wtab32)));
    return BLD_OK;
}

// large dynamic shared memory (the most a B200 block may opt into), and the largest
// shared-memory carveout so the per-SM block count is set by the kernel's real footprint
#define BLD_SET(K)                                                                                 \
    do {                                                                                           \
        CUDA_TRY(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)); \
        CUDA_TRY(cudaFuncSetAttribute(K, cudaFuncAttributePreferredSharedMemoryCarveout,           \
                                      cudaSharedmemCarveoutMaxShared));                            \
    } while (0)

}  // namespace bld
