// Device pieces that the flow stages and the measurement share.
#pragma once

#include "kernels.cuh"
#include "launch.cuh"

namespace glac {

// Force of a link from its staple sum.  FP64 forms only the part of U A that
// enters; in FP32 at 80 registers the full product was the faster one.
template <typename T> __device__ __forceinline__ AH8<T> flow_force(const M3<T> &U, const M3<T> &A) {
    if constexpr (sizeof(T) == 4) return project_ah(mul(U, A));
    else return project_ah_mul(U, A);
}

// The end of a flow stage for one link with force Z: the RK3 combination, the
// stored force, U' = exp(M) U.
template <typename T, int KIND, int STAGE>
__device__ __forceinline__ void flow_update(const M3<T> &U, const AH8<T> &Z, const LinkField<T> &out,
                                            const ForceField<T> &zf, T alpha, T beta, int mu, int p, int s) {
    AH8<T> M;
    if (STAGE == 0) {
        M = ah_scale(alpha, Z);
        zf.store(mu, p, s, Z);
    } else {
        const AH8<T> W = zf.load(mu, p, s);
        M = ah_axpby(alpha, Z, beta, W);
        if (STAGE == 1) zf.store(mu, p, s, M);
    }
    chain_release();
    if (KIND == EXP_MORNINGSTAR) {
        // U' = U + (exp(M) - 1) U: the small product first, one rounding at |U|
        out.store(mu, p, s, mul_plus_right(expm_morningstar<T, true>(M), U));
    } else {
        out.store(mu, p, s, mul(expm<T>(KIND, M), U));
    }
}

// (C - C^+) made traceless, in the 8-real form: diagonal 2 i Im C_ii minus a
// third of its trace, off-diagonal C_ij - conj(C_ji).  Linear in C.
template <typename T> __device__ __forceinline__ AH8<T> proj_ah8(const M3<T> &C) {
    AH8<T> F;
    const T two = T(2);
    const T tr = (C(0, 0).im + C(1, 1).im + C(2, 2).im) * T(2.0 / 3.0);
    F.a = two * C(0, 0).im - tr;
    F.d = two * C(1, 1).im - tr;
    F.b = cx(C(0, 1).re - C(1, 0).re, C(0, 1).im + C(1, 0).im);
    F.c = cx(C(0, 2).re - C(2, 0).re, C(0, 2).im + C(2, 0).im);
    F.e = cx(C(1, 2).re - C(2, 1).re, C(1, 2).im + C(2, 1).im);
    return F;
}
template <typename T> __device__ __forceinline__ AH8<T> ah_add(const AH8<T> &X, const AH8<T> &Y) {
    AH8<T> Z;
    Z.a = X.a + Y.a;
    Z.d = X.d + Y.d;
    Z.b = X.b + Y.b;
    Z.c = X.c + Y.c;
    Z.e = X.e + Y.e;
    return Z;
}

// plane index of (a, b), a < b: 01 0, 02 1, 03 2, 12 3, 13 4, 23 5
__host__ __device__ constexpr int plane_of(int a, int b) { return a == 0 ? b - 1 : (a == 1 ? b + 1 : 5); }
// the planes link direction mu takes (nu, or -1)
__device__ __forceinline__ bool meas_takes(int mu, int nu) {
    return (mu == 0 && (nu == 1 || nu == 2)) || (mu == 1 && (nu == 2 || nu == 3)) || (mu == 2 && nu == 3) ||
           (mu == 3 && nu == 0);
}

template <typename T> __device__ __forceinline__ AH8<T> ah_neg_if(const AH8<T> &F, bool neg) {
    return neg ? ah_scale(T(-1), F) : F;
}

// P(A B), negated where neg: twice project_ah of the product, with its sign turned
// (FP64; FP32 forms the product, as flow_force).
template <typename T> __device__ __forceinline__ AH8<T> clover_part(const M3<T> &A, const M3<T> &B, bool neg) {
    if constexpr (sizeof(T) == 4) return ah_neg_if(proj_ah8(mul(A, B)), neg);
    else return ah_scale(neg ? T(2) : T(-2), project_ah_mul(A, B));
}

// Re Tr(F G) for traceless anti-Hermitian F, G in the 8-real form:
//   -[a a' + d d' + (a+d)(a'+d')] - 2 Re(b b'* + c c'* + e e'*)
template <typename T>
__device__ __forceinline__ T retr_ah(const AH8<T> &F, const AH8<T> &G) {
    T diag = fmaR(F.a, G.a, F.d * G.d);
    diag = fmaR(F.a + F.d, G.a + G.d, diag);
    T off = fmaR(F.b.re, G.b.re, F.b.im * G.b.im);
    off = fmaR(F.c.re, G.c.re, off);
    off = fmaR(F.c.im, G.c.im, off);
    off = fmaR(F.e.re, G.e.re, off);
    off = fmaR(F.e.im, G.e.im, off);
    return -(diag + off + off);
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// en += sum ReTr(F F) and qt = -[ReTr(F_01 F_23) + ReTr(F_02 F_31) + ReTr(F_03 F_12)]
// (F_31 = -F_13) of a site's six projected clovers.
template <typename T> __device__ __forceinline__ void clover_sums(const AH8<T> F[6], double &en, double &qt) {
    qt = -((double)retr_ah(F[0], F[5]) - (double)retr_ah(F[1], F[4]) + (double)retr_ah(F[2], F[3]));
#pragma unroll
    for (int pl = 0; pl < 6; pl++) en += (double)retr_ah(F[pl], F[pl]);
}

template <typename T>
__device__ __forceinline__ void combine_site(const Geom &g, const CloverParts<T> &cp, int p, int s, double &plaq,
                                             double &en, double &qt) {
    AH8<T> F[6];
#pragma unroll
    for (int pl = 0; pl < 6; pl++) F[pl] = ah_add(cp.ah.load(2 * pl, p, s), cp.ah.load(2 * pl + 1, p, s));
#pragma unroll
    for (int mu = 0; mu < 4; mu++) plaq += (double)cp.plaq[(mu * 2 + p) * g.Vh + s];
    clover_sums(F, en, qt);
}

// Block sums of the three per-thread values in a fixed order (warp shuffles,
// then the warps in order) into partial[3 b .. 3 b + 2] = (plaq, energy, q).
__device__ __forceinline__ void obs_block_reduce(double plaq, double en, double qt, double *partial, int b) {
    __shared__ double sh[3][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    plaq = warp_sum_d(plaq);
    en = warp_sum_d(en);
    qt = warp_sum_d(qt);
    if (lane == 0) { sh[0][wid] = plaq; sh[1][wid] = en; sh[2][wid] = qt; }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        double a = 0.0, e = 0.0, q = 0.0;
        for (int w = 0; w < nw; w++) { a += sh[0][w]; e += sh[1][w]; q += sh[2][w]; }
        partial[3 * b] = a;
        partial[3 * b + 1] = e;
        partial[3 * b + 2] = q;
    }
}

// out = [plaq, topc, energy, topct[Nt]] with the reference's normalisations
// (mastersamplertopcxyz.cpp:13-16, :363-383).
// Per-slice sums by warps (slice t on warp t mod W; lane l adds the partials
// l, l+32, ..., then a fixed xor-shuffle tree), the slices then in order by one
// thread: the same operations in the same order every call.
__device__ __forceinline__ void obs_finalize_body(int Nt, int nb, int V, const double *partial, double *out) {
    __shared__ double sp[1024], se[1024], sq[1024];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int t = warp; t < Nt; t += nwarps) {
        double a = 0.0, e = 0.0, q = 0.0;
        const double *pt = partial + 3 * (size_t)t * 2 * nb;
        for (int k = lane; k < 2 * nb; k += 32) {
            a += pt[3 * k];
            e += pt[3 * k + 1];
            q += pt[3 * k + 2];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            e += __shfl_xor_sync(0xffffffffu, e, o);
            q += __shfl_xor_sync(0xffffffffu, q, o);
        }
        if (lane == 0) { sp[t] = a; se[t] = e; sq[t] = q; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double qfac = 1.0 / (16 * 16 * M_PI * M_PI);
        double a = 0.0, e = 0.0, q = 0.0;
        for (int t = 0; t < Nt; t++) { a += sp[t]; e += se[t]; q += sq[t]; }
        out[0] = a / (18.0 * (double)V);
        out[1] = q * qfac;
        out[2] = e / (double)V;
        for (int t = 0; t < Nt; t++) out[3 + t] = sq[t] * qfac;
    }
}
}  // namespace glac
