// x passes with in-place two-pass line transforms (bld_row::k_adv_row, bld_row::k_sgs_x).
//
// A block owns NR y rows and walks up a z chunk; per layer the packed lines of
// its rows go to the physical domain, the products are formed point by point
// with the previous layer's values in registers, and the results go back.  A
// line of P = A B points lives in ONE shared-memory buffer through both
// transforms, as A blocks of B places, so every pass reads and writes the same
// addresses from the same thread:
//   inverse 1: task j (< B) gathers the packed spectrum n = j + B t (t < A), radix-A
//              DFT over t, output q to block q, place j;
//   inverse 2: task q (< A) multiplies its block by W_P^(j q), radix-B DFT over j,
//              output m in place: the value at x = q + A m sits in block q, place m;
//   products:  pointwise, the same places of the lines of a row;
//   forward 1: task q: radix-B DFT of its block, times W_P^(q k'), in place;
//   forward 2: task k' (< B) gathers place k' of all blocks, radix-A DFT:
//              X[k' + B k2], k2 < A, in registers.  The partner X[P - k] of the
//              two-lines-in-one unpacking is held by the lane of task B - k' of the
//              same warp: two or four shuffles per mode fetch it, and the modes
//              k <= k1max go straight to global memory.
// The input rows of layer j + 1 are fetched by 1-d TMA bulk copies into the one
// staging area as soon as inverse pass 1 of layer j has read it.
//
// What bounds it: the transforms, not the bytes.  k_adv_x2 / k_sgs_x2 hold pass-1
// outputs, physical lines, forward lines and two staging areas apart (113 to 195 KB a
// block, one or two blocks of four to ten warps per SM) and stall on their block
// barriers (41 % of samples).  One buffer for both directions and one staging area
// leave two to eight independent blocks per SM, four barriers per layer instead of
// five, and no spectra in shared memory.  Measured (us per launch, before -> now):
// advection 192^2 x 96 double 238 -> 181, single 130 -> 99; 512^2 x 64 single
// 944 -> 466; 128^2 x 64 single 45 -> 35; Smagorinsky 256^2 x 64 double 584 -> 287,
// 512^2 x 64 single 920 -> 600, 128^2 x 64 single 71 -> 47.  Now shared-memory
// wavefronts (48 to 64 % of peak) and issue slots (32 to 62 %) share the time.
#pragma once

#include "bld_dft.cuh"
#include "bld_tma.cuh"
#include "bld_xargs.cuh"

namespace bld_row {

__host__ __device__ constexpr int xr_al(int b) { return (b + 127) / 128 * 128; }
// elements between the blocks of a line: odd, so that tasks on consecutive blocks
// meet no bank conflicts; and between lines
__host__ __device__ constexpr int xr_blk(int B) { return B | 1; }
__host__ __device__ constexpr int xr_line(int A, int B) { return A * xr_blk(B); }

// packed spectrum value Z[n] of the lines a + i b from half spectra: `lo` takes
// A + i B, the mirrored half conj(A) + i conj(B); FFTW's c2r convention at DC
template <typename R>
__device__ __forceinline__ cplx<R> xr_pack(cplx<R> va, cplx<R> vb, bool dc, bool lo) {
    if (dc) return mk<R>(va.x, vb.x);
    return lo ? mk<R>(va.x - vb.y, va.y + vb.x) : mk<R>(va.x + vb.y, vb.x - va.y);
}

template <typename T>
__device__ __forceinline__ T xr_shfl(T v, int lane) {
    return __shfl_sync(0xffffffffu, v, lane);
}

// inverse pass 2 / forward pass 1 on one block of a line, in place
template <typename R, int A, int B, int DIR>
__device__ __forceinline__ void xr_block(cplx<R>* blk, const cplx<R>* tw, int q) {
    using C = cplx<R>;
    C x[B];
#pragma unroll
    for (int t = 0; t < B; ++t) x[t] = blk[t];
    if (DIR > 0) {
#pragma unroll
        for (int t = 1; t < B; ++t) x[t] = c_tw<DIR>(x[t], tw[t * A + q]);
    }
    dft<R, B, DIR>(x);
    if (DIR < 0) {
#pragma unroll
        for (int t = 1; t < B; ++t) x[t] = c_tw<DIR>(x[t], tw[t * A + q]);
    }
#pragma unroll
    for (int t = 0; t < B; ++t) blk[t] = x[t];
}

// ------------------------------------------------------------------- advection
// dynamic shared memory: barrier, twiddles, 6 terms x NR rows, lines
__host__ __device__ constexpr int ar_smem(int A, int B, int K1, int csz, int NR, bool sepf) {
    return 128 + xr_al(A * B * csz) + xr_al(6 * NR * K1 * csz) + xr_al(3 * NR * xr_line(A, B) * csz) +
           (sepf ? xr_al((NR + NR / 2) * xr_line(A, B) * csz) : 0);
}

// values carried from one layer to the next at one point
template <typename R>
struct AdvCarry {
    R w, o1, o2, c;   // w, vort1, vort2 on the I layer below and vort2 u - vort1 v there
};

// grid (ceil(P2 / NR), nchunks, members), block T threads.  SEPF: the forward lines have
// their own buffer, so the stores of layer j share a barrier interval with inverse
// pass 1 of layer j + 1.  Needs 3 k1max < P (middle third of the spectrum empty)
// where A is a multiple of 3.
template <typename R, int A, int B, int NR, int T, int MINB, bool SEPF>
__global__ void __launch_bounds__(T, MINB) k_adv_row(XArgs a) {
    using C = cplx<R>;
    constexpr int P = A * B, NLI = 3 * NR, NLF = NR + NR / 2, LS = xr_line(A, B), BS = xr_blk(B);
    constexpr bool TH = A % 3 == 0;
    constexpr int PPT = (NR * P + T - 1) / T;
    constexpr int KM = TH ? A / 3 : (A + 1) / 2;   // k2 of the modes k' + B k2 <= k1max
    constexpr int csz = (int)sizeof(C);
    constexpr int LW = 32 / B;   // lines per warp in forward pass 2
    static_assert(NR % 2 == 0 && B <= 32 && T % 32 == 0, "shape");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    C* tw = reinterpret_cast<C*>(smem_raw + 128);
    const C* twg = reinterpret_cast<const C*>(a.tw);
    for (int i = threadIdx.x; i < P; i += T) tw[i] = twg[(i / A) * (i % A)];   // [t][q]: W_P^(t q)
    grid_wait();   // every block, whether it has work or not
    const int n3 = a.g.n3, k1max = a.g.k1max, K1 = a.g.K1;
    const int m = a.m0 + blockIdx.z;
    BLD_SKIP_INACTIVE(a, m);
    const int y0 = blockIdx.x * NR;
    const int z0 = blockIdx.y * a.zchunk, z1 = min(n3, z0 + a.zchunk);
    if (z0 >= z1) return;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    unsigned char* p = smem_raw + 128;
    p += xr_al(P * csz);
    C* stage = reinterpret_cast<C*>(p);
    p += xr_al(6 * NR * K1 * csz);
    C* Ln = reinterpret_cast<C*>(p);
    p += xr_al(NLI * LS * csz);
    C* Fw = SEPF ? reinterpret_cast<C*>(p) : Ln;
    const C* Min = reinterpret_cast<const C*>(a.min) + (long long)m * a.min_mstride;
    C* Mout = reinterpret_cast<C*>(a.mout) + (long long)m * a.mout_mstride;
    const int nr = min(NR, a.P2 - y0);   // rows of this block (even); the others are not stored
    const unsigned row_bytes = (unsigned)(nr * K1 * csz);
    // staged slots: u, v, vort3 (C); w, vort1, vort2 (I) = mixed terms 0, 1, 5, 2, 3, 4
    auto issue = [&](int j) {
        const int nslots = (j < n3 - 1) ? 6 : 3;
        mbar_arrive_expect_tx(bar, nslots * row_bytes);
        for (int r = 0; r < nslots; ++r) {
            const int t = r < 2 ? r : (r == 2 ? 5 : r - 1);
            bulk_load(stage + (size_t)r * NR * K1, mrow(Min, a, t, j, y0), row_bytes, bar);
        }
    };
    const int jb = max(0, z0 - 1);
    const long long wait_limit = *a.wait_limit;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_async_shared();
        issue(jb);
    }
    AdvCarry<R> cy[PPT];
#pragma unroll
    for (int i = 0; i < PPT; ++i) cy[i] = AdvCarry<R>{R(0), R(0), R(0), R(0)};
    __syncthreads();

    for (int j = jb; j < z1; ++j) {
        const bool hasI = (j < n3 - 1);
        const bool arrived = mbar_wait_bounded(bar, (j - jb) & 1, wait_limit);
        // ---- inverse pass 1: lines 3 r + p = pairs (u, v), (vort3, w), (vort1, vort2)
        for (int task = threadIdx.x; task < NLI * B; task += T) {
            const int L = task / B, jt = task % B;
            const int r = L / 3, pp = L - 3 * r;
            if (pp == 2 && !hasI) continue;
            const C* ra = stage + (2 * pp * NR + r) * K1;
            const C* rb = ra + NR * K1;
            const bool okb = pp != 1 || hasI;
            C x[A];
#pragma unroll
            for (int t = 0; t < A; ++t) {
                const int n = jt + B * t;
                if (TH && t >= A / 3 && t < A - A / 3) {
                    x[t] = mk<R>(R(-0.0), R(-0.0));   // -0: adding it folds away
                    continue;
                }
                const bool lo = TH ? t < A / 3 : n <= k1max, hi = n >= P - k1max;
                const int idx = lo ? n : P - n;
                C va = mk<R>(R(0), R(0)), vb = mk<R>(R(0), R(0));
                if ((TH && lo) ? n <= k1max : (lo || hi)) {
                    va = ra[idx];
                    if (okb) vb = rb[idx];
                }
                x[t] = xr_pack<R>(va, vb, t == 0 && jt == 0, lo);
            }
            dft<R, A, +1>(x);
#pragma unroll
            for (int q = 0; q < A; ++q) Ln[L * LS + q * BS + jt] = x[q];
        }
        // a block whose wait expired stops here (uniformly), after its copies have landed
        if (__syncthreads_or(!arrived)) {
            if (threadIdx.x == 0) {
                atomicOr(a.flag + m, BLD_FLAG_TIMEOUT);
                mbar_wait_bounded(bar, (j - jb) & 1);
            }
            return;
        }
        if (threadIdx.x == 0 && j + 1 < z1) {
            fence_async_shared();
            issue(j + 1);
        }
        // ---- inverse pass 2
        for (int task = threadIdx.x; task < NLI * A; task += T) {
            const int L = task / A, q = task - L * A;
            if (L % 3 == 2 && !hasI) continue;
            xr_block<R, A, B, +1>(Ln + L * LS + q * BS, tw, q);
        }
        __syncthreads();
        // ---- products at one point of one row
        const bool emitC = (j >= z0);
        const bool emitI = (j >= z0) && (j >= 1);
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            const int idx = threadIdx.x + T * i;
            if (idx < NR * P) {
                const int r = idx / P, s = idx - r * P;
                const int pos = s + (BS - B) * (s / B);
                C* l0 = Ln + 3 * r * LS + pos;
                const C c0 = l0[0], c1 = l0[LS];
                const C c2 = hasI ? l0[2 * LS] : mk<R>(R(0), R(0));
                const R u = c0.x, v = c0.y, o3 = c1.x;
                const R w = hasI ? c1.y : R(0);
                const R q1 = c2.x, q2 = c2.y;
                AdvCarry<R>& k = cy[i];
                // w vanishes at both boundaries: the carried and the new w are zero
                // there (:180-201)
                const R adv1 = o3 * v - R(0.5) * (k.o2 * k.w + q2 * w);
                const R adv2 = R(0.5) * (k.o1 * k.w + q1 * w) - o3 * u;
                // adv3 on I layer j - 1 (:206)
                const R adv3 = R(0.5) * ((k.o2 * u - k.o1 * v) + k.c);
                if (SEPF) {
                    Fw[r * LS + pos] = mk<R>(adv1, adv2);
                    reinterpret_cast<R*>(Fw + (NR + r / 2) * LS + pos)[r & 1] = adv3;
                } else {
                    l0[0] = mk<R>(adv1, adv2);
                    l0[LS].x = adv3;
                }
                k.w = w;
                k.o1 = q1;
                k.o2 = q2;
                k.c = q2 * u - q1 * v;
            }
        }
        __syncthreads();
        // forward lines 0..NR-1: (adv1, adv2) of C layer j; NR..: adv3 of two rows, I layer j - 1
        const int lf0 = emitC ? 0 : NR, lf1 = emitI ? NLF : NR;
        // ---- forward pass 1
        for (int task = threadIdx.x; task < (lf1 - lf0) * A; task += T) {
            const int L = lf0 + task / A, q = task % A;
            C* blk;
            if (SEPF) blk = Fw + L * LS + q * BS;
            else blk = Fw + (L < NR ? 3 * L : 6 * (L - NR) + 1) * LS + q * BS;
            if (!SEPF && L >= NR) {
                C x[B];
#pragma unroll
                for (int t = 0; t < B; ++t) x[t] = mk<R>(blk[t].x, blk[t + 3 * LS].x);
                dft<R, B, -1>(x);
#pragma unroll
                for (int t = 1; t < B; ++t) x[t] = c_tw<-1>(x[t], tw[t * A + q]);
#pragma unroll
                for (int t = 0; t < B; ++t) blk[t] = x[t];
            } else {
                xr_block<R, A, B, -1>(blk, tw, q);
            }
        }
        __syncthreads();
        // ---- forward pass 2, unpacking and the store of the modes
        for (int l0 = lf0 + (threadIdx.x >> 5) * LW; l0 < lf1; l0 += (T / 32) * LW) {
            const int lane = threadIdx.x & 31, g = lane / B, kp = lane % B;
            const int L = g < LW && l0 + g < lf1 ? l0 + g : l0;
            const bool ok = L == l0 + g && (L < NR ? L : 2 * (L - NR)) < nr;
            const C* src = Fw + (SEPF ? L : (L < NR ? 3 * L : 6 * (L - NR) + 1)) * LS + kp;
            C x[A];
#pragma unroll
            for (int t = 0; t < A; ++t) x[t] = src[t * BS];
            dft<R, A, -1>(x);
            const int partner = g < LW && kp ? lane + B - 2 * kp : lane;
            C *oa, *ob;
            if (L < NR) {
                oa = mrow_w(Mout, a, 0, j, y0 + L) + kp;
                ob = mrow_w(Mout, a, 1, j, y0 + L) + kp;
            } else {
                oa = mrow_w(Mout, a, 2, j - 1, y0 + 2 * (L - NR)) + kp;
                ob = oa + K1;
            }
#pragma unroll
            for (int k2 = 0; k2 < KM; ++k2) {
                C Zr = mk<R>(xr_shfl(x[A - 1 - k2].x, partner), xr_shfl(x[A - 1 - k2].y, partner));
                if (kp == 0) Zr = x[(A - k2) % A];
                const C Zk = x[k2];
                if (ok && kp + B * k2 <= k1max) {
                    oa[B * k2] = mk<R>((Zk.x + Zr.x) * R(0.5), (Zk.y - Zr.y) * R(0.5));
                    ob[B * k2] = mk<R>((Zk.y + Zr.y) * R(0.5), (Zr.x - Zk.x) * R(0.5));
                }
            }
        }
        if (!SEPF) __syncthreads();
    }
}

// ----------------------------------------------------------------- Smagorinsky
// The x derivatives of the inputs and of the stresses are factors i k1 2 pi / L1 of
// the modes this kernel reads and writes, so only u, v, w and their y derivatives
// come in (six mixed terms: u, v, w, u_2, v_2, w_2) and per velocity component only
// d1 tau_i1 + d3 tau_i3 and tau_i2 go out (six: the three sums, then tau12, tau22,
// tau23).
//
// d3 tau_i3 shares a line with tau_i1, so both are rounded at the size of the larger, and
// tau_i1 is multiplied by its wavenumber afterwards.  Near a wall d3 tau exceeds the
// stresses by the vertical resolution; scaled by a power of two next to one over the
// largest wavenumber on its way through the transform it adds nothing to the rounding of
// d1 tau_i1 (vel1 of a right-hand side at 128^2 x 64, error against 64 bits relative to
// separate lines: 1.077 without the scale and 1.000 with it in double, 1.074 and 1.000 in
// single precision; 64^2 x 64 stretched, single, 1.191 and 1.000; scales from an eighth to
// four times this one are as good).  The sums go out times 2 d3_scale, the stresses times 2
// (the halves of the two-lines-in-one unpacking), and the forward y pass takes that back.
__host__ __device__ constexpr int sr_lines_in(int NR) { return 4 * NR + (NR + 1) / 2; }
// dynamic shared memory: barrier, twiddles, x wavenumbers, 6 terms x NR rows, lines
__host__ __device__ constexpr int sr_smem(int A, int B, int K1, int csz, int NR) {
    return 128 + xr_al(A * B * csz) + xr_al(K1 * csz / 2) + xr_al(6 * NR * K1 * csz) +
           xr_al(sr_lines_in(NR) * xr_line(A, B) * csz) + xr_al(4 * NR * xr_line(A, B) * csz);
}

// values carried from one layer to the next at one point: velocities and strains of
// the C layer below, S13, S23 and the eddy viscosity of the I layer below it, and
// tau33 of the C layer before
template <typename R>
struct SgsRow {
    R u, v, w, w1, w2, s11, s22, s33, s12, s13, s23, ev, t33;
};

// layer-dependent factors of one step of the z walk (uniform over the block)
template <typename R>
struct SgsLayer {
    R ac_j, ai_b, li_b, lc_c;   // alpha_c[j], alpha_i[j-1], li[j-1], lc[j-1]
    R ac_c, ai_c;               // d3_alpha_c[j-1], d3_alpha_i[j-2]
};

// The Smagorinsky model at one point when C layer j enters, as sgs_point
// (src/processes/static_smagorinsky.jl:129-249), with the three stresses of the I
// nodes and d3 tau33 all given on I layer j - 2: o = (tau11, d3 tau13, tau12,
// d3 tau23, tau13, d3 tau33, tau22, tau23), the d3 terms times d3_scale.
template <typename R>
__device__ __forceinline__ void sgs_row_point(const XArgs& a, const SgsLayer<R>& y, int j, int n3, bool hasC, R fs_lo,
                                              R fs_hi, R ft_lo, R ft_hi, R wlo, R u, R v, R u1, R u2, R v1, R v2, R w,
                                              R w1, R w2, SgsRow<R>& k, R (&o)[8]) {
    const int c = j - 1;
    R s11 = 0, s22 = 0, s33 = 0, s12 = 0;
    if (hasC) {
        const R wb = (j == 0) ? wlo : k.w;
        s33 = -y.ac_j * wb + y.ac_j * w;
        s11 = u1;
        s22 = v2;
        s12 = (u2 + v1) * R(0.5);
    }
    // I layer j - 1
    R s13 = 0, s23 = 0, ev = 0;
    if (j >= 1 && j <= n3 - 1) {
        s13 = ((-y.ai_b * k.u + y.ai_b * u) + k.w1) * R(0.5);
        s23 = ((-y.ai_b * k.v + y.ai_b * v) + k.w2) * R(0.5);
        R si = R(2) * (s13 * s13) + R(2) * (s23 * s23);
        R t;
        t = k.s11 + s11; si += t * t * R(0.25);
        t = k.s22 + s22; si += t * t * R(0.25);
        t = k.s33 + s33; si += t * t * R(0.25);
        t = k.s12 + s12; si += t * t * R(0.5);
        ev = sqrt(R(2) * si) * y.li_b;
    }
    const R sg13 = R(-2) * ev * s13, sg23 = R(-2) * ev * s23;
#pragma unroll
    for (int q = 0; q < 8; ++q) o[q] = 0;
    if (j >= 1) {
        // C layer c = j - 1
        R scc = k.s11 * k.s11 + k.s22 * k.s22 + k.s33 * k.s33 + R(2) * (k.s12 * k.s12);
        const R p13 = R(-2) * k.ev * k.s13, p23 = R(-2) * k.ev * k.s23;   // stresses on I layer c - 1
        R below13 = p13, below23 = p23, above13 = sg13, above23 = sg23;
        if (c == 0 || c == n3 - 1) {   // wall-adjacent layers: dynamic values are not interpolated (:195-200,:245-249)
            const bool lo = c == 0;
            const R uh = sqrt(k.u * k.u + k.v * k.v);
            if (lo ? a.dyn_lo : a.dyn_hi) {
                const R f = lo ? fs_lo : fs_hi;
                R d = k.u * f;
                scc += R(2) * (d * d);
                d = k.v * f;
                scc += R(2) * (d * d);
            } else {
                R d = lo ? s13 : k.s13;
                scc += d * d * R(0.5);
                d = lo ? s23 : k.s23;
                scc += d * d * R(0.5);
            }
            if (lo) {
                below13 = a.dyn_lo ? ft_lo * k.u * uh : R(0);
                below23 = a.dyn_lo ? ft_lo * k.v * uh : R(0);
            } else {
                above13 = a.dyn_hi ? ft_hi * k.u * uh : R(0);
                above23 = a.dyn_hi ? ft_hi * k.v * uh : R(0);
            }
        } else {
            R d = k.s13 + s13;
            scc += d * d * R(0.5);
            d = k.s23 + s23;
            scc += d * d * R(0.5);
        }
        const R evc = sqrt(R(2) * scc) * y.lc_c;
        o[0] = R(2) * evc * k.s11;
        o[2] = R(2) * evc * k.s12;
        o[6] = R(2) * evc * k.s22;
        const R sg33 = R(-2) * evc * k.s33;
        o[1] = y.ac_c * below13 - y.ac_c * above13;
        o[3] = y.ac_c * below23 - y.ac_c * above23;
        if (c >= 1) o[5] = y.ai_c * k.t33 - y.ai_c * sg33;
        o[4] = -p13;
        o[7] = -p23;
        k.t33 = sg33;
    }
    k.s13 = s13; k.s23 = s23; k.ev = ev;
    if (hasC) {
        k.s11 = s11; k.s22 = s22; k.s33 = s33; k.s12 = s12;
        k.u = u; k.v = v; k.w = w; k.w1 = w1; k.w2 = w2;
    }
}

// grid (P2 / NR, nchunks, members), block T threads; P1 = A B = 2 k1max + 2
template <typename R, int A, int B, int NR, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) k_sgs_x(XArgs a) {
    using C = cplx<R>;
    constexpr int P = A * B, NLI = sr_lines_in(NR), NLF = 4 * NR, LS = xr_line(A, B), BS = xr_blk(B);
    constexpr int PPT = (NR * P + T - 1) / T;
    constexpr int csz = (int)sizeof(C);
    constexpr int LW = 32 / B;   // lines per warp in forward pass 2
    static_assert((NR == 1 || NR % 2 == 0) && B <= 32 && A % 2 == 0 && T % 32 == 0, "shape");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    C* tw = reinterpret_cast<C*>(smem_raw + 128);
    const C* twg = reinterpret_cast<const C*>(a.tw);
    for (int i = threadIdx.x; i < P; i += T) tw[i] = twg[(i / A) * (i % A)];   // [t][q]: W_P^(t q)
    grid_wait();   // every block, whether it has work or not
    const int n3 = a.g.n3, k1max = a.g.k1max, K1 = a.g.K1;
    const int m = a.m0 + blockIdx.z;
    BLD_SKIP_INACTIVE(a, m);
    const int y0 = blockIdx.x * NR;
    const int z0 = blockIdx.y * a.zchunk, z1 = min(n3, z0 + a.zchunk);
    if (z0 >= z1) return;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    unsigned char* p = smem_raw + 128;
    p += xr_al(P * csz);
    R* dk = reinterpret_cast<R*>(p);
    p += xr_al(K1 * csz / 2);
    C* stage = reinterpret_cast<C*>(p);
    p += xr_al(6 * NR * K1 * csz);
    C* Ln = reinterpret_cast<C*>(p);
    p += xr_al(NLI * LS * csz);
    C* Fw = reinterpret_cast<C*>(p);   // the forward lines have a buffer of their own
    const C* Min = reinterpret_cast<const C*>(a.min) + (long long)m * a.min_mstride;
    C* Mout = reinterpret_cast<C*>(a.mout) + (long long)m * a.mout_mstride;
    const double* lcm = a.lc + (long long)m * n3;
    const double* lim = a.li + (long long)m * (n3 - 1);
    const R fs_lo = (R)a.wall[4 * m + 0], fs_hi = (R)a.wall[4 * m + 1];
    const R ft_lo = (R)a.wall[4 * m + 2], ft_hi = (R)a.wall[4 * m + 3];
    const R wlo = (R)a.w_lo, whi = (R)a.w_hi;
    const R d3_scale = sizeof(R) == 4 ? (R)a.d3_scale32 : (R)a.d3_scale;
    const unsigned row_bytes = (unsigned)(NR * K1 * csz);
    const long long wait_limit = *a.wait_limit;
    // staged slots: u, v, u_2, v_2 (C); w, w_2 (I, below the top layer) = mixed terms 0, 1, 3, 4, 2, 5
    auto issue = [&](int j) {
        const int nslots = (j <= n3 - 2) ? 6 : 4;
        mbar_arrive_expect_tx(bar, nslots * row_bytes);
        for (int s = 0; s < nslots; ++s)
            bulk_load(stage + (size_t)s * NR * K1, mrow(Min, a, (0x524310 >> (4 * s)) & 0xF, j, y0), row_bytes, bar);
    };
    const int jb = max(0, z0 - 2);
    const int jend = min(n3, z1 + 1);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_async_shared();
        issue(jb);   // jb <= z0 <= n3 - 1
    }
    for (int i = threadIdx.x; i < K1; i += T) dk[i] = (R)a.d1[i];
    SgsRow<R> cy[PPT];
#pragma unroll
    for (int i = 0; i < PPT; ++i) cy[i] = SgsRow<R>{};
    __syncthreads();

    for (int j = jb; j <= jend; ++j) {
        const bool hasC = (j <= n3 - 1), hasI = (j <= n3 - 2);
        if (hasC) {
            const bool arrived = mbar_wait_bounded(bar, (j - jb) & 1, wait_limit);
            // ---- inverse pass 1: lines 4 r + q = pairs (u, v), (u_1, u_2), (v_1, v_2),
            // (w_1, w); then w_2 of two rows per line
            for (int task = threadIdx.x; task < NLI * B; task += T) {
                const int L = task / B, jt = task % B;
                const int r = L < 4 * NR ? L / 4 : 2 * (L - 4 * NR), q = L < 4 * NR ? L % 4 : 4;
                if (q >= 3 && !hasI) continue;
                const C* ra = stage + (((0x54100 >> (4 * q)) & 0xF) * NR + r) * K1;
                const C* rb = q < 4 ? stage + (((0x4321 >> (4 * q)) & 0xF) * NR + r) * K1 : ra + K1;
                const bool da = q >= 1 && q <= 3, okb = q < 4 || NR > 1;
                C x[A];
#pragma unroll
                for (int t = 0; t < A; ++t) {
                    const int n = jt + B * t;
                    const bool lo = t < A / 2;
                    const int idx = lo ? n : P - n;
                    C va = mk<R>(R(0), R(0)), vb = mk<R>(R(0), R(0));
                    if (t != A / 2 || jt != 0) {   // n = P / 2 is not resolved
                        va = ra[idx];
                        if (okb) vb = rb[idx];
                        if (da) {
                            const R d = dk[idx];
                            va = mk<R>(-d * va.y, d * va.x);
                        }
                    }
                    x[t] = xr_pack<R>(va, vb, t == 0 && jt == 0, lo);
                }
                dft<R, A, +1>(x);
#pragma unroll
                for (int q2 = 0; q2 < A; ++q2) Ln[L * LS + q2 * BS + jt] = x[q2];
            }
            // a block whose wait expired stops here (uniformly), after its copies have landed
            if (__syncthreads_or(!arrived)) {
                if (threadIdx.x == 0) {
                    atomicOr(a.flag + m, BLD_FLAG_TIMEOUT);
                    mbar_wait_bounded(bar, (j - jb) & 1);
                }
                return;
            }
            if (threadIdx.x == 0 && j + 1 <= min(jend, n3 - 1)) {
                fence_async_shared();
                issue(j + 1);
            }
            // ---- inverse pass 2
            for (int task = threadIdx.x; task < NLI * A; task += T) {
                const int L = task / A, q = task - L * A;
                if (!hasI && (L >= 4 * NR || L % 4 == 3)) continue;
                xr_block<R, A, B, +1>(Ln + L * LS + q * BS, tw, q);
            }
            __syncthreads();
        } else {
            __syncthreads();   // the forward lines of the layer below have been read
        }
        const int c = j - 1;   // C layer completed at this step
        const bool doC = (j >= 1) && (c >= z0) && (c < z1);
        const bool doI = (j >= 2) && (j - 2 >= z0) && (j - 2 < z1) && (j - 2 <= n3 - 2);
        SgsLayer<R> ly;
        ly.ac_j = hasC ? (R)__ldg(a.alpha_c + j) : R(0);
        ly.ai_b = (j >= 1 && hasC) ? (R)__ldg(a.alpha_i + j - 1) : R(0);
        ly.li_b = (j >= 1 && hasC) ? (R)lim[j - 1] : R(0);
        ly.lc_c = j >= 1 ? (R)lcm[j - 1] : R(0);
        ly.ac_c = j >= 1 ? (R)__ldg(a.d3_alpha_c + j - 1) : R(0);
        ly.ai_c = j >= 2 ? (R)__ldg(a.d3_alpha_i + j - 2) : R(0);
        // ---- the model at one point of one row
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            const int idx = threadIdx.x + T * i;
            if (idx < NR * P) {
                const int r = idx / P, s = idx - r * P;
                const int pos = s + (BS - B) * (s / B);
                const C* l0 = Ln + 4 * r * LS + pos;
                R u = 0, v = 0, u1 = 0, u2 = 0, v1 = 0, v2 = 0, w = whi, w1 = 0, w2 = 0;
                if (hasC) {
                    const C c0 = l0[0], c1 = l0[LS], c2 = l0[2 * LS];
                    u = c0.x; v = c0.y; u1 = c1.x; u2 = c1.y; v1 = c2.x; v2 = c2.y;
                    if (hasI) {
                        const C c3 = l0[3 * LS];
                        w1 = c3.x; w = c3.y;
                        w2 = reinterpret_cast<const R*>(Ln + (4 * NR + r / 2) * LS + pos)[r & 1];
                    }
                }
                R o[8];
                sgs_row_point<R>(a, ly, j, n3, hasC, fs_lo, fs_hi, ft_lo, ft_hi, wlo, u, v, u1, u2, v1, v2, w, w1, w2,
                                 cy[i], o);
                if (doC || doI) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) Fw[(4 * r + q) * LS + pos] = mk<R>(o[2 * q], o[2 * q + 1]);
                }
            }
        }
        if (!doC && !doI) {
            __syncthreads();   // the model is done with the lines
            continue;
        }
        __syncthreads();
        // ---- forward pass 1
        for (int task = threadIdx.x; task < NLF * A; task += T) {
            const int L = task / A, q = task - L * A;
            xr_block<R, A, B, -1>(Fw + L * LS + q * BS, tw, q);
        }
        __syncthreads();
        // ---- forward pass 2, unpacking and the store of the modes
        for (int l0 = (threadIdx.x >> 5) * LW; l0 < NLF; l0 += (T / 32) * LW) {
            const int lane = threadIdx.x & 31, g = lane / B, kp = lane % B;
            const bool ok = g < LW && l0 + g < NLF;
            const int L = ok ? l0 + g : l0;
            const int r = L / 4, q = L % 4;
            const C* src = Fw + L * LS + kp;
            C x[A];
#pragma unroll
            for (int t = 0; t < A; ++t) x[t] = src[t * BS];
            dft<R, A, -1>(x);
            const int partner = ok && kp ? lane + B - 2 * kp : lane;
            // first result: d1 tau + d3 tau of lines 0..2 (times 2 d3_scale), tau22 of line 3;
            // second: tau12, tau23 (all times 2)
            const bool first = ok && (q == 2 ? doI : doC), second = ok && (q == 1 ? doC : q == 3 && doI);
            C* o1 = mrow_w(Mout, a, q < 3 ? q : 4, q == 2 ? j - 2 : c, y0 + r) + kp;
            C* o2 = mrow_w(Mout, a, q == 1 ? 3 : 5, q == 1 ? c : j - 2, y0 + r) + kp;
#pragma unroll
            for (int k2 = 0; k2 < A / 2; ++k2) {
                C Zr = mk<R>(xr_shfl(x[A - 1 - k2].x, partner), xr_shfl(x[A - 1 - k2].y, partner));
                if (kp == 0) Zr = x[(A - k2) % A];
                const C Zk = x[k2];
                const C va = mk<R>(Zk.x + Zr.x, Zk.y - Zr.y);
                const C vb = mk<R>(Zk.y + Zr.y, Zr.x - Zk.x);
                if (kp + B * k2 <= k1max) {
                    const R d = dk[kp + B * k2] * d3_scale;
                    if (first) o1[B * k2] = q < 3 ? mk<R>(vb.x - d * va.y, vb.y + d * va.x) : va;
                    if (second) o2[B * k2] = q == 1 ? va : vb;
                }
            }
        }
    }
}

}  // namespace bld_row
