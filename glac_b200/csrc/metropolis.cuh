// A Metropolis proposal and its accept weight, shared by the sub-sweep kernels.
#pragma once

#include "kernels.cuh"

namespace glac {

// Proposal uniform (h + 1/2) 2^-16 - 1/2 of a 16-bit word without a conversion
// instruction: 2^23 + h read from its bit pattern, minus 2^23, gives h exactly;
// (2h + 1 - 2^16) 2^-17 has at most 17 significant bits, so the FMA is exact.
__device__ __forceinline__ float u_sym16f(uint32_t h) {
    const float hf = __uint_as_float(0x4B000000u | h) - 8388608.f;
    return __fmaf_rn(hf, 1.f / 65536.f, 0.5f / 65536.f - 0.5f);
}
// FP64 the same way: 2^52 + h from its bit pattern (FP64 conversions run on the
// special-function pipe).
__device__ __forceinline__ double u32_to_double(uint32_t h) {
    return __hiloint2double(0x43300000, (int)h) - 4503599627370496.0;
}
__device__ __forceinline__ double u_sym16d(uint32_t h) {
    return __fma_rn(u32_to_double(h), 1.0 / 65536.0, 0.5 / 65536.0 - 0.5);
}
template <typename T> __device__ __forceinline__ T proposal_uniform(uint32_t h);
template <> __device__ __forceinline__ double proposal_uniform<double>(uint32_t h) { return u_sym16d(h); }
template <> __device__ __forceinline__ float proposal_uniform<float>(uint32_t h) { return u_sym16f(h); }

// Accept uniform in [0, 1): 53 bits for FP64; for FP32 the 23 high bits of word 6
// as the mantissa of a float in [1, 2), minus 1 (no conversion instruction).
template <typename T> __device__ __forceinline__ T accept_uniform(uint32_t w6, uint32_t w7);
template <> __device__ __forceinline__ double accept_uniform<double>(uint32_t w6, uint32_t w7) {
    // (w6 2^21 + (w7 >> 11)) 2^-53: 53 bits, so the FMA does not round
    return __fma_rn(u32_to_double(w6), 2097152.0, u32_to_double(w7 >> 11)) * 1.1102230246251565e-16;
}
template <> __device__ __forceinline__ float accept_uniform<float>(uint32_t w6, uint32_t) {
    return __uint_as_float(0x3F800000u | (w6 >> 9)) - 1.f;
}

template <typename T>
__device__ __forceinline__ void su2_near_unity(T u0, T u1, T u2, T u3, T eps, T sq1me, bool flips, T out[4]);
// x0 = sign(u0) sqrt(1 - eps^2), x = eps u / |u|, normalised
// (GLAC/math/matrices/su3matrixgenerator.h:202-243); without flips x0 > 0.
// FP64: |x|^2 = (1 - eps^2) + eps^2 is 1 to a few ulp whatever u is, so the
// normalisation 1 / sqrt(q) is its first-order term 3/2 - q/2 (the next one is
// below 1e-30), and u / |u| takes one reciprocal square root: the eight
// divisions and two square roots of the formula as written had been most of a
// hit's FP64 operations (four sweeps of 16^3 x 32 on B200: 2.57 ms with them and
// with converted uniforms, 1.52 ms so).
template <>
__device__ __forceinline__ void su2_near_unity<double>(double u0, double u1, double u2, double u3, double eps,
                                                       double sq1me, bool flips, double out[4]) {
    const double x0 = (flips && u0 < 0.0) ? -sq1me : sq1me;
    const double sc = eps * rsqrt(u1 * u1 + u2 * u2 + u3 * u3);
    const double x1 = u1 * sc, x2 = u2 * sc, x3 = u3 * sc;
    const double inv = fma(-0.5, x0 * x0 + x1 * x1 + x2 * x2 + x3 * x3, 1.5);
    out[0] = x0 * inv; out[1] = x1 * inv; out[2] = x2 * inv; out[3] = x3 * inv;
}
// FP32: the same construction with reciprocal square roots in place of the
// square roots and divisions (which load the special-function pipe).
template <>
__device__ __forceinline__ void su2_near_unity<float>(float u0, float u1, float u2, float u3, float eps, float sq1me,
                                                      bool flips, float out[4]) {
    const float x0 = (flips && u0 < 0.f) ? -sq1me : sq1me;
    const float sc = eps * rsqrtf(u1 * u1 + u2 * u2 + u3 * u3);
    const float x1 = u1 * sc, x2 = u2 * sc, x3 = u3 * sc;
    const float inv = rsqrtf(x0 * x0 + x1 * x1 + x2 * x2 + x3 * x3);
    out[0] = x0 * inv; out[1] = x1 * inv; out[2] = x2 * inv; out[3] = x3 * inv;
}

// X = R S T with the SU(2) elements [[x0 + i x3, x2 + i x1], [-x2 + i x1, x0 - i x3]]
// embedded in the (12), (13), (23) blocks; zero blocks skipped.  inverse -> X^+.
template <typename T>
__device__ __forceinline__ M3<T> rst_matrix(const T r[4], const T s[4], const T t[4], bool inverse) {
    const Cx<T> r00 = cx(r[0], r[3]), r01 = cx(r[2], r[1]), r10 = cx(-r[2], r[1]), r11 = cx(r[0], -r[3]);
    const Cx<T> s00 = cx(s[0], s[3]), s01 = cx(s[2], s[1]), s10 = cx(-s[2], s[1]), s11 = cx(s[0], -s[3]);
    const Cx<T> t00 = cx(t[0], t[3]), t01 = cx(t[2], t[1]), t10 = cx(-t[2], t[1]), t11 = cx(t[0], -t[3]);
    // R S = [[r00 s00, r01, r00 s01], [r10 s00, r11, r10 s01], [s10, 0, s11]]
    const Cx<T> a0 = r00 * s00, a2 = r00 * s01, b0 = r10 * s00, b2 = r10 * s01;
    M3<T> X;
    X(0, 0) = a0;
    X(1, 0) = b0;
    X(2, 0) = s10;
    X(0, 1) = cmac(r01 * t00, a2, t10);
    X(1, 1) = cmac(r11 * t00, b2, t10);
    X(2, 1) = s11 * t10;
    X(0, 2) = cmac(r01 * t01, a2, t11);
    X(1, 2) = cmac(r11 * t01, b2, t11);
    X(2, 2) = s11 * t11;
    return inverse ? dagger(X) : X;
}

template <typename T>
__device__ __forceinline__ void draw_proposal(uint32_t k0, uint32_t k1, uint32_t link_id, uint32_t sweep,
                                              uint32_t stream_id, int hit, T eps, T sq1me, bool flips, M3<T> &X,
                                              T &r) {
    uint32_t w[8];
#pragma unroll
    for (int call = 0; call < 2; call++) {
        U4 c = {(uint32_t)(2 * hit + call), link_id, sweep, stream_id};
        U4 o = philox4x32_10(c, k0, k1);
        w[4 * call] = o.x; w[4 * call + 1] = o.y; w[4 * call + 2] = o.z; w[4 * call + 3] = o.w;
    }
    T su[3][4];
#pragma unroll
    for (int b = 0; b < 3; b++) {
        T u[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int k = 4 * b + c;
            const uint32_t word = w[k >> 1];
            u[c] = proposal_uniform<T>((k & 1) ? (word >> 16) : (word & 0xFFFFu));
        }
        su2_near_unity<T>(u[0], u[1], u[2], u[3], eps, sq1me, flips, su[b]);
    }
    X = rst_matrix<T>(su[0], su[1], su[2], (w[7] & 1u) == 0u);
    r = accept_uniform<T>(w[6], w[7]);
}

// exp(-dS) in the working precision (compared with accept_uniform<T>)
template <typename T> __device__ __forceinline__ T accept_weight(T dS);
template <> __device__ __forceinline__ double accept_weight<double>(double dS) { return exp(-dS); }
template <> __device__ __forceinline__ float accept_weight<float>(float dS) { return expf(-dS); }

template <typename T>
__device__ __forceinline__ T delta_s(const M3<T> &U, const M3<T> &Up, const M3<T> &A, T mfac) {
    M3<T> D = Up;
    sub_from(D, U);
    return retr_mul(D, A) * mfac;
}

// Small lattices: a link's staple and hits over several warps (metro_split.cu).
bool metropolis_splits(const Geom &g);
template <typename T>
void launch_metropolis_split(const Geom &g, const LinkField<T> &L, int mu, int p, T mfac, T eps, T sq1me, int nhits,
                             uint32_t k0, uint32_t k1, uint32_t sweep, uint32_t stream_id, unsigned long long *acc,
                             const Proposal &P, float beta, cudaStream_t st);

}  // namespace glac
