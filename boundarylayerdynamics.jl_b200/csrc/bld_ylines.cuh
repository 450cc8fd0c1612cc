// y passes on NL neighbouring k1 lines per block (k_inv_yl, k_fwd_yl).
//
// The two-pass transforms of bld_ypass2.cuh (P2 = A B, thread tid works on line
// tid % NL, task tid / NL, one buffer of shared memory in place), for every
// P2 = A B of the codelet sizes, with
//  * the structure of the padded spectrum fixed at compile time: with the 3/2 rule
//    (band 1) the middle third of the inverse transform's inputs is zero and of the
//    forward transform's outputs unused, on the default grid (band 2) only the Nyquist
//    row is; the zeros are -0.0, which the first butterflies fold away;
//  * pass-1 outputs at an odd stride where a row of lines is shorter than the 128 bytes
//    of the banks, and the twiddles of pass 2 as [s][j], so that the lanes of a warp
//    read neighbouring entries;
//  * the Laplacian of the forward epilogue as three weights of the window of layers,
//    the same for the whole block (ghost layers included), instead of the boundary
//    forms worked out per output.
//
// What bounds them: the latency of the global loads, at 40 % of DRAM throughput or less;
// the more warps are resident the better, so the registers are held as low as the larger
// radix allows.  The forward epilogue took two thirds of that pass's instructions.
// Measured (us per launch, k_inv_y2 / k_fwd_y2 -> here): inverse 512^2 x 32 single
// 768 points 186 -> 162, 128^2 x 256 single 192 points 81 -> 66, 192^2 x 96 288 points
// single 70 -> 62, double 104 -> 100, 128^2 x 512 double 128 points 156 -> 136; forward
// 192^2 x 96 288 points double 153 -> 107, single 113 -> 79; 512^2 x 32 single
// 768 points 237 -> 180, 512 points with two line sets 277 -> 239; 128^2 x 256 single
// 192 points 113 -> 76.
#pragma once

#include "bld_kernels.cuh"
#include "bld_ypass2.cuh"

namespace bld_yl {

// elements between pass-1 tasks' outputs: A rows of NL lines, made odd where a row is
// shorter than the banks
__host__ __device__ constexpr int task_stride(int A, int NL, int csz) { return NL * csz % 128 ? (A | 1) : A; }
__host__ __device__ constexpr int smem_bytes(int A, int B, int NL, int csz, int sets) {
    return (A * B + sets * task_stride(A, NL, csz) * B * NL) * csz;
}

// inverse pass 1 for term kind OP: gather the padded spectral line straight from the
// state, radix-A DFT, store
template <typename R, int A, int B, int NL, int BAND, int OP>
__device__ __forceinline__ void inv_pass1(const InvYArgs& a, const double2* S, int f, int z, int k1, bool ok, int j,
                                          cplx<R>* buf) {
    using C = cplx<R>;
    constexpr int P = A * B, AP = task_stride(A, NL, (int)sizeof(C));
    const Geo& g = a.g;
    const int F = g.F, n3 = g.n3, k2max = g.k2max, shift = P - g.K2;
    const double2* Su = S + (long long)z * F;
    const double2* Sv = Su + (long long)n3 * F;
    const double2* Sw = Sv + (long long)n3 * F;
    const double2* Sf = S + ((long long)f * n3 + z) * F;
    const double e1 = ok ? __ldg(a.d1 + k1) : 0.0;
    const double al = (OP == T_VORT1 || OP == T_VORT2) ? __ldg(a.alpha_i + z) : 0.0;
    C x[A];
#pragma unroll
    for (int t = 0; t < A; ++t) {
        const int p = j + B * t;
        if (BAND == 1 && t >= A / 3 && t < A - A / 3) {
            x[t] = mk<R>(R(-0.0), R(-0.0));
            continue;
        }
        int jj;
        bool in;
        if (BAND == 1) {
            jj = t < A / 3 ? p : p - shift;
            in = t < A / 3 ? p <= k2max : p >= P - k2max;
        } else if (BAND == 2) {
            jj = t < A / 2 ? p : p - shift;
            in = t != A / 2 || j != 0;
        } else {
            jj = p <= k2max ? p : p - shift;
            in = p <= k2max || p >= P - k2max;
        }
        double2 v = make_double2(0.0, 0.0);
        if (ok && in) {
            const double e2 = (OP == T_D2 || OP == T_VORT1 || OP == T_VORT3) ? __ldg(a.d2 + jj) : 0.0;
            v = y2_term<OP>(Sf, Su, Sv, Sw, F, jj * g.K1 + k1, e1, e2, al);
        }
        x[t] = mk<R>((R)v.x, (R)v.y);
    }
    dft<R, A, +1>(x);
#pragma unroll
    for (int q = 0; q < A; ++q) buf[(j * AP + q) * NL] = x[q];
}

// grid (nterms * members, ceil(K1 / NL), n3), block max(A, B) NL threads, dynamic smem
// smem_bytes(.., 1).  SGS: the terms u, v, w and their y derivatives; else u, v, w and
// the vorticity.
template <typename R, int A, int B, int NL, int MINB, int BAND, bool SGS>
__global__ void __launch_bounds__((A > B ? A : B) * NL, MINB) k_inv_yl(InvYArgs a) {
    using C = cplx<R>;
    constexpr int P = A * B, AP = task_stride(A, NL, (int)sizeof(C)), T = (A > B ? A : B) * NL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* buf = tw + P;
    const C* twg = reinterpret_cast<const C*>(a.tw);
    for (int i = threadIdx.x; i < P; i += T) tw[i] = twg[(i / A) * (i % A)];   // [s][j]: W_P^(j s)
    grid_wait();   // every block, whether it has work or not
    const int t = blockIdx.x % a.nterms, m = a.m0 + blockIdx.x / a.nterms;
    BLD_SKIP_INACTIVE(a, m);
    const int z = blockIdx.z;
    const int nz = a.isI[t] ? a.g.n3 - 1 : a.g.n3;
    if (z >= nz) return;
    const int op = a.op[t], f = a.fld[t];
    const int K1 = a.g.K1;
    const int l = threadIdx.x % NL, j = threadIdx.x / NL;
    const int k1 = blockIdx.y * NL + l;
    const bool ok = k1 < K1;
    const double2* S = a.state + (long long)m * a.g.mstride;
    if (B >= A || j < B) {
        if constexpr (SGS) {
            if (op == T_DIRECT) inv_pass1<R, A, B, NL, BAND, T_DIRECT>(a, S, f, z, k1, ok, j, buf + l);
            else inv_pass1<R, A, B, NL, BAND, T_D2>(a, S, f, z, k1, ok, j, buf + l);
        } else {
            switch (op) {
                case T_DIRECT: inv_pass1<R, A, B, NL, BAND, T_DIRECT>(a, S, f, z, k1, ok, j, buf + l); break;
                case T_VORT1: inv_pass1<R, A, B, NL, BAND, T_VORT1>(a, S, f, z, k1, ok, j, buf + l); break;
                case T_VORT2: inv_pass1<R, A, B, NL, BAND, T_VORT2>(a, S, f, z, k1, ok, j, buf + l); break;
                default: inv_pass1<R, A, B, NL, BAND, T_VORT3>(a, S, f, z, k1, ok, j, buf + l); break;
            }
        }
    }
    __syncthreads();
    if (A < B && j >= A) return;
    C x[B];
#pragma unroll
    for (int s = 0; s < B; ++s) x[s] = buf[(s * AP + j) * NL + l];
#pragma unroll
    for (int s = 1; s < B; ++s) x[s] = c_tw<+1>(x[s], tw[s * A + j]);
    dft<R, B, +1>(x);
    if (!ok) return;
    C* out = reinterpret_cast<C*>(a.mixed) + (long long)m * a.mixed_mstride +
             ((long long)(t * a.g.n3 + z) * P + j) * K1 + k1;
#pragma unroll
    for (int q = 0; q < B; ++q) out[(long long)(A * q) * K1] = x[q];
}

// The linear terms of a field at layer z (the same as linear_terms, for a whole block) as
// weights of the window of layers w0 .. w0 + 2:
//   nu ((e0 + c0 coef) W0 + (e1 + c1 coef) W1 + (e2 + c2 coef) W2 + all) (+ mean for the
// mean mode), coef = DD1 + DD2 - ab - bc and c = 1 for layer z itself
// (src/processes/molecular_diffusion.jl:57-72, src/boundary_conditions.jl:254-359,
// src/processes/sources.jl:32-35).
struct LinWeights {
    double e0, e1, e2, c0, c1, c2, ab, bc, nu, all, mean;
};
__device__ __forceinline__ LinWeights lin_weights(const Geo& g, const Linear& L, int f, int z, int w0, int m) {
    LinWeights w;
    w.e0 = w.e1 = w.e2 = w.ab = w.bc = w.nu = w.all = w.mean = 0.0;
    const int r0 = z - w0;
    w.c0 = r0 == 0;
    w.c1 = r0 == 1;
    w.c2 = r0 == 2;
    if (L.diff_on[f]) {
        const int n = (f == 2) ? g.n3 - 1 : g.n3;
        double A, B, Cc;
        if (f != 2) {
            A = L.alpha_ext[z];
            B = L.alpha_c[z];
            Cc = L.alpha_ext[z + 1];
        } else {
            A = L.alpha_c[z];
            B = L.alpha_i[z];
            Cc = L.alpha_c[z + 1];
        }
        w.ab = A * B;
        w.bc = B * Cc;
        w.nu = L.nu[f];
        auto add = [&](int r, double v) {
            if (r == 0) w.e0 += v;
            else if (r == 1) w.e1 += v;
            else w.e2 += v;
        };
        // layer z - 1, or the ghost layer below by extrapolation from the three next to the wall
        if (z > 0) {
            add(r0 - 1, w.ab);
        } else if (f == 2) {
            w.all += w.ab * L.bc_val[2][0];   // Dirichlet values of w enter every mode
        } else if (L.bc_kind[f][0] == 0) {
            add(0, w.ab * -3.0);
            add(1, w.ab);
            add(2, w.ab * (-1.0 / 5.0));
            w.mean += w.nu * (w.ab * (16.0 * L.bc_val[f][0] / 5.0));
        } else {
            add(0, w.ab * (21.0 / 23.0));
            add(1, w.ab * (3.0 / 23.0));
            add(2, w.ab * (-1.0 / 23.0));
            w.mean -= w.nu * (w.ab * (24.0 * L.bc_diff[f][0] / 23.0));
        }
        // layer z + 1, or the ghost layer above
        if (z < n - 1) {
            add(r0 + 1, w.bc);
        } else if (f == 2) {
            w.all += w.bc * L.bc_val[2][1];
        } else if (L.bc_kind[f][1] == 0) {
            add(2, w.bc * -3.0);
            add(1, w.bc);
            add(0, w.bc * (-1.0 / 5.0));
            w.mean += w.nu * (w.bc * (16.0 * L.bc_val[f][1] / 5.0));
        } else {
            add(2, w.bc * (21.0 / 23.0));
            add(1, w.bc * (3.0 / 23.0));
            add(0, w.bc * (-1.0 / 23.0));
            w.mean += w.nu * (w.bc * (24.0 * L.bc_diff[f][1] / 23.0));
        }
    }
    if (L.src_on[f]) w.mean += L.src[3 * m + f];
    return w;
}

// grid (fields * members, ceil(K1 / NL), n3), block max(A, B) NL threads, dynamic smem
// smem_bytes(.., SETS).  SETS = 1: one mixed term per field; 2: and one under D2, on a
// second set of lines.  Modes 0 and 1 of FwdYArgs, rates or fused stage values.
template <typename R, int A, int B, int NL, int MINB, int BAND, int SETS>
__global__ void __launch_bounds__((A > B ? A : B) * NL, MINB) k_fwd_yl(FwdYArgs a) {
    using C = cplx<R>;
    constexpr int P = A * B, AP = task_stride(A, NL, (int)sizeof(C)), T = (A > B ? A : B) * NL, NJ = T / NL;
    constexpr int SB = B * AP * NL;   // elements of one line set
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* buf = tw + P;
    const C* twg = reinterpret_cast<const C*>(a.tw);
    for (int i = threadIdx.x; i < P; i += T) tw[i] = twg[(i / A) * (i % A)];   // [s][j]: W_P^(j s)
    grid_wait();   // every block, whether it has work or not
    const int fi = blockIdx.x % a.fields, m = a.m0 + blockIdx.x / a.fields;
    BLD_SKIP_INACTIVE(a, m);
    const int f = a.field0 + fi;
    const int z = blockIdx.z;
    const Geo& g = a.g;
    const int nz = (f == 2) ? g.n3 - 1 : g.n3;
    if (z >= nz) return;
    const int K1 = g.K1;
    const int l = threadIdx.x % NL, j = threadIdx.x / NL;
    const int k1 = blockIdx.y * NL + l;
    const bool ok = k1 < K1;
    const C* base = reinterpret_cast<const C*>(a.mout) + (long long)m * a.mout_mstride + k1;
#pragma unroll 1
    for (int set = 0; set < SETS; ++set) {
        if (j < B) {
            const C* src = base + ((long long)(a.c[fi][set].term * g.n3 + z) * P + j) * K1;
            C x[A];
#pragma unroll
            for (int t = 0; t < A; ++t) x[t] = ok ? src[(long long)(B * t) * K1] : mk<R>(0, 0);
            dft<R, A, -1>(x);
#pragma unroll
            for (int q = 0; q < A; ++q) buf[set * SB + (j * AP + q) * NL + l] = x[q];
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int set = 0; set < SETS; ++set) {
        if (j < A) {
            C* b = buf + set * SB + j * NL + l;
            C x[B];
#pragma unroll
            for (int s = 0; s < B; ++s) x[s] = b[s * AP * NL];
#pragma unroll
            for (int s = 1; s < B; ++s) x[s] = c_tw<-1>(x[s], tw[s * A + j]);
            dft<R, B, -1>(x);
            // X[j + A q] in place of X1[j + A q]; the middle third is not resolved
#pragma unroll
            for (int q = 0; q < B; ++q)
                if (BAND != 1 || B % 3 || q < B / 3 || q >= B - B / 3) b[q * AP * NL] = x[q];
        }
    }
    __syncthreads();
    // ---- epilogue: truncation, scaling, D2, linear terms or the rate so far, stage update
    const int K2 = g.K2, k2max = g.k2max;
    const long long fo = (long long)m * a.du_mstride + fld_off(g, f) + (long long)z * g.F;
    double2* du = a.du + fo;
    const double2* Sf = a.state ? a.state + (long long)m * g.mstride + fld_off(g, f) : nullptr;
    const int w0 = lin_window_start(z, nz);
    bool bad = false;
    auto epilogue = [&](auto mode_c, auto fuse_c) {
        constexpr int MODE = decltype(mode_c)::value;   // 1: with the linear terms, 0: added to du
        constexpr int FZ = decltype(fuse_c)::value;     // 0: the rate; 1: su, state and rate; 2: state and rate
        const double2* su = FZ == 1 ? a.su + fo : nullptr;
        double2* so = FZ ? a.sout + fo : du;
        LinWeights w;
        double dd1 = 0.0;
        const bool three = nz >= 3;
        if constexpr (MODE == 1) {
            w = lin_weights(g, a.lin, f, z, w0, m);
            dd1 = ok ? __ldg(a.lin.DD1 + k1) : 0.0;
        }
        if (!ok) return;
        // the state may take the non-coherent path: it was complete before the x pass began,
        // and this kernel is launched once that has
        const double2* S0 = MODE == 1 ? Sf + (long long)w0 * g.F + k1 : nullptr;
        const double2* Sz = MODE != 1 && FZ != 0 ? Sf + (long long)z * g.F + k1 : nullptr;
        for (int jj = j; jj < K2; jj += NJ) {
            const int o = jj * K1;
            double2 W0, W1, W2, U, t;
            if constexpr (MODE == 1) {
                W0 = __ldg(S0 + o);
                W1 = __ldg(S0 + g.F + o);
                W2 = three ? __ldg(S0 + 2 * g.F + o) : make_double2(0.0, 0.0);
            } else {
                W0 = du[k1 + o];
                if constexpr (FZ != 0) t = __ldg(Sz + o);
            }
            if constexpr (FZ == 1) U = su[k1 + o];
            const int p = jj <= k2max ? jj : P - (K2 - jj);
            const int slot = AP == A ? p : (p / A) * AP + p % A;
            const C X = buf[slot * NL + l];
            double vx = (double)X.x * a.inv_a, vy = (double)X.y * a.inv_a;
            if constexpr (SETS == 2) {
                const C Y = buf[SB + slot * NL + l];
                const double d = __ldg(a.d2 + jj);
                vx += -d * ((double)Y.y * a.inv_b);
                vy += d * ((double)Y.x * a.inv_b);
            }
            if constexpr (MODE == 1) {
                const double coef = ((dd1 + __ldg(a.lin.DD2 + jj)) - w.ab) - w.bc;
                const double f0 = w.e0 + w.c0 * coef, f1 = w.e1 + w.c1 * coef, f2 = w.e2 + w.c2 * coef;
                double lx = w.nu * (((f0 * W0.x + f1 * W1.x) + f2 * W2.x) + w.all);
                const double ly = w.nu * ((f0 * W0.y + f1 * W1.y) + f2 * W2.y);
                if (jj == 0 && k1 == 0) lx += w.mean;
                vx += lx;
                vy += ly;
                if constexpr (FZ != 0) t = w.c0 != 0.0 ? W0 : (w.c1 != 0.0 ? W1 : W2);
            } else {
                vx += W0.x;
                vy += W0.y;
            }
            if (!(isfinite(vx) && isfinite(vy))) bad = true;
            if constexpr (FZ == 1) {
                vx = (a.st_cu * U.x + a.st_ct * t.x + a.st_cd * vx) * a.st_inv;
                vy = (a.st_cu * U.y + a.st_ct * t.y + a.st_cd * vy) * a.st_inv;
            } else if constexpr (FZ == 2) {   // Euler stage: state + dt rate (src/ODEMethods.jl:101)
                vx = t.x + a.st_cd * vx;
                vy = t.y + a.st_cd * vy;
            }
            so[k1 + o] = make_double2(vx, vy);
        }
    };
    using I0 = std::integral_constant<int, 0>;
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    const int fz = a.fuse ? (a.su ? 1 : 2) : 0;
    // a field with one term per rate is the first (or only) to write it; with two line sets
    // it adds to another's, or is the only process
    if (a.mode == 1) {
        if (fz == 0) epilogue(I1{}, I0{});
        else if (fz == 1) epilogue(I1{}, I1{});
        else epilogue(I1{}, I2{});
    } else {
        if (fz == 0) epilogue(I0{}, I0{});
        else if (fz == 1) epilogue(I0{}, I1{});
        else epilogue(I0{}, I2{});
    }
    if (a.check && bad) atomicOr(a.flag + m, BLD_FLAG_NONFINITE);
}

}  // namespace bld_yl
