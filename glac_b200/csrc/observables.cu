// The stand-alone measurement of a single lattice: plaquette, clover energy and
// topological charge, their densities, and the Weinberg operator.
//
// As in the measurement inside flow stage 0 (kernels.cu), the clover of plane
// (mu, nu) at n comes from the staple pieces of the links mu at n and n - mu:
// with W = S_up - S_low at n, F(n) = P(U W)(n) + P(W U)(n - mu).  One kernel, a
// thread per plane and site, forms W and both parts, 5.7 products where a site's
// own four leaves take 10 (12 with each leaf from its four links), and six times
// the threads; the second adds the two parts of each of a site's six planes and
// reduces.  The parts lie in the context's second field and its force, which
// hold nothing between flow steps.
#include "kernels.cuh"
#include "flow_body.cuh"
#include "launch.cuh"

#include <stdexcept>

namespace glac {

template <typename T>
__device__ __forceinline__ void clover_parts_body(const Geom &g, const LinkField<T> &L, const PlaneParts<T> &parts,
                                                  int bx) {
    const int plane = bx % 12, pl = plane >> 1, p = plane & 1, q = p ^ 1;
    const int s = (bx / 12) * 128 + threadIdx.x;
    if (s >= g.Vh) return;
    // (mu, nu) of planes 01 02 03 12 13 23
    const int mu = pl < 3 ? 0 : pl < 5 ? 1 : 2, nu = pl < 3 ? pl + 1 : pl < 5 ? pl - 1 : 3;
    const Site n = site_from_ps(g, p, s);
    const int f_mu = step_offset(g, n, mu, +1), b_nu = step_offset(g, n, nu, -1);
    const int s_mu = (n.lex + f_mu) >> 1, s_nup = (n.lex + step_offset(g, n, nu, +1)) >> 1;
    const int s_num = (n.lex + b_nu) >> 1, s_diag = (n.lex + f_mu + b_nu) >> 1;
    M3<T> W = mul_nd(mul_nd(L.load(nu, q, s_mu), L.load(mu, q, s_nup)), L.load(nu, p, s));
    parts.plaq[(pl * 2 + p) * g.Vh + s] = retr_mul(L.load(mu, p, s), W);
    asm volatile("" ::: "memory");
    sub_mul(W, mul_dd(L.load(nu, p, s_diag), L.load(mu, q, s_num)), L.load(nu, q, s_num));
    asm volatile("" ::: "memory");
    chain_release();
    parts.store(2 * pl, p, s, clover_part(L.load(mu, p, s), W, false));
    asm volatile("" ::: "memory");
    parts.store(2 * pl + 1, q, s_mu, clover_part(W, L.load(mu, p, s), false));
}
template <typename T, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) k_clover_parts(Geom g, LinkField<T> L, PlaneParts<T> parts) {
    chain_wait();
    clover_parts_body<T>(g, L, parts, blockIdx.x);
}

// What a measurement keeps of each site besides the sums.
enum ObsMode { OBS_SUMS = 0, OBS_DENSITY = 1, OBS_WEINBERG = 2 };

// Weinberg operator (GLAC/observables/supersampler.cpp:298-496) from the six
// clovers of a site: for nu = 1..3 and (rho, sigma) the cyclic complement of nu,
//   w = -sum ReTr[(sum_{lambda != nu} G_{0 lambda} G_{nu lambda}) G_{rho sigma}],
// G_{b a} = G_{a b}^+ for the orientations the reference does not store (:421-433).
template <typename T> __device__ __forceinline__ double weinberg_site(const AH8<T> F[6]) {
    // G0[nu] = G_{0 nu}; Gc[nu] = G_{rho sigma}: G_23, G_31 = -G_13, G_12
    AH8<T> G0[4], Gc[4];
    G0[1] = F[0]; G0[2] = F[1]; G0[3] = F[2];
    Gc[1] = F[5]; Gc[2] = ah_scale(T(-1), F[4]); Gc[3] = F[3];
    double w = 0.0;
#pragma unroll
    for (int nu = 1; nu < 4; nu++) {
        M3<T> acc;
        set_zero(acc);
#pragma unroll
        for (int lam = 1; lam < 4; lam++) {
            if (lam == nu) continue;
            // (nu, lam) in {(1,2), (2,3), (3,1)} is stored as Gc[the third index]; the reverse is its dagger
            const M3<T> m = ah_to_m3(Gc[6 - nu - lam]);
            acc_mul(acc, ah_to_m3(G0[lam]), lam == nu % 3 + 1 ? m : dagger(m));
        }
        w -= (double)retr_mul(acc, ah_to_m3(Gc[nu]));
    }
    return w;
}

// Block b covers Bv sites of one (t, parity) half slice, so its sums are
// partials of that slice.  dq, de (OBS_DENSITY): the per-site fields of
// LatticeActionChargeDensity (latticeactionchargedensity.cpp:169-306) in
// lexicographic order, dq = -(1/(16^2 pi^2)) sum ReTr(C_0nu C_rhosigma) and
// de = sum ReTr(C C) (unnormalised).
template <typename T, ObsMode MODE>
__global__ void __launch_bounds__(256) k_plane_combine(Geom g, PlaneParts<T> parts, int nb, int Bv, double *partial,
                                                       double *dq, double *de) {
    chain_wait();
    const int b = blockIdx.x;
    const int t = b / (2 * nb);
    const int p = (b / nb) & 1;
    const int j = b % nb;
    const int half_slice = g.Vh / g.N[3];
    const bool valid = (int)threadIdx.x < Bv;
    const int s = t * half_slice + j * Bv + (valid ? (int)threadIdx.x : 0);
    double plaq = 0.0, en = 0.0, qt = 0.0, wt = 0.0;
    if (valid) {
        AH8<T> F[6];
#pragma unroll
        for (int pl = 0; pl < 6; pl++) F[pl] = ah_add(parts.load(2 * pl, p, s), parts.load(2 * pl + 1, p, s));
#pragma unroll
        for (int pl = 0; pl < 6; pl++) plaq += (double)parts.plaq[(pl * 2 + p) * g.Vh + s];
        clover_sums(F, en, qt);
        if (MODE == OBS_WEINBERG) wt = weinberg_site(F);
        if (MODE == OBS_DENSITY) {
            const int lex = site_from_ps(g, p, s).lex;
            dq[lex] = qt * (1.0 / (16 * 16 * M_PI * M_PI));
            de[lex] = en;
        }
    }
    if (MODE != OBS_WEINBERG) {
        obs_block_reduce(plaq, en, qt, partial, b);
        return;
    }
    __shared__ double sh[4][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    plaq = warp_sum_d(plaq);
    en = warp_sum_d(en);
    qt = warp_sum_d(qt);
    wt = warp_sum_d(wt);
    if (lane == 0) { sh[0][wid] = plaq; sh[1][wid] = en; sh[2][wid] = qt; sh[3][wid] = wt; }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        double a = 0.0, e = 0.0, q = 0.0, w = 0.0;
        for (int k = 0; k < nw; k++) { a += sh[0][k]; e += sh[1][k]; q += sh[2][k]; w += sh[3][k]; }
        partial[4 * b] = a;
        partial[4 * b + 1] = e;
        partial[4 * b + 2] = q;
        partial[4 * b + 3] = w;
    }
}

// One measurement per block: rows of 3 (2 nb Nt) partials in, rows of 3 + Nt out.
__global__ void k_obs_finalize(int Nt, int nb, int V, const double *partial, double *out) {
    chain_wait();
    obs_finalize_body(Nt, nb, V, partial + (size_t)blockIdx.x * 6 * nb * Nt, out + (size_t)blockIdx.x * (3 + Nt));
}
void launch_obs_finalize(const Geom &g, int nb, int rows, const double *partial, double *out, cudaStream_t st) {
    if (g.N[3] > 1024) throw std::invalid_argument("Nt > 1024 not supported by the observable reduction");
    launch_chained(k_obs_finalize, rows, 1024, st, g.N[3], nb, g.V, partial, out);
}

// out = [plaq, topc, energy, weinberg, topct[Nt], weinbergt[Nt]], the Weinberg factor
// 2 * 8 * 8 / (3 * 16^3) (supersampler.cpp:13)
__global__ void k_weinberg_finalize(int Nt, int nb, int V, const double *partial, double *out) {
    chain_wait();
    __shared__ double sp[1024], se[1024], sq[1024], sw[1024];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int t = warp; t < Nt; t += nwarps) {
        double a = 0.0, e = 0.0, q = 0.0, w = 0.0;
        const double *pt = partial + 4 * (size_t)t * 2 * nb;
        for (int k = lane; k < 2 * nb; k += 32) {
            a += pt[4 * k];
            e += pt[4 * k + 1];
            q += pt[4 * k + 2];
            w += pt[4 * k + 3];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            e += __shfl_xor_sync(0xffffffffu, e, o);
            q += __shfl_xor_sync(0xffffffffu, q, o);
            w += __shfl_xor_sync(0xffffffffu, w, o);
        }
        if (lane == 0) { sp[t] = a; se[t] = e; sq[t] = q; sw[t] = w; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double qfac = 1.0 / (16 * 16 * M_PI * M_PI), wfac = 2 * 8.0 * 8.0 / (3 * 16 * 16 * 16);
        double a = 0.0, e = 0.0, q = 0.0, w = 0.0;
        for (int t = 0; t < Nt; t++) { a += sp[t]; e += se[t]; q += sq[t]; w += sw[t]; }
        out[0] = a / (18.0 * (double)V);
        out[1] = q * qfac;
        out[2] = e / (double)V;
        out[3] = w * wfac;
        for (int t = 0; t < Nt; t++) {
            out[4 + t] = sq[t] * qfac;
            out[4 + Nt + t] = sw[t] * wfac;
        }
    }
}

template <typename T>
static void clover_parts(const Geom &g, const LinkField<T> &L, const PlaneParts<T> &parts, int variant,
                         cudaStream_t st) {
    if (g.N[3] > 1024) throw std::invalid_argument("Nt > 1024 not supported by the observable reduction");
    const int grid = 12 * ((g.Vh + 127) / 128);
    if constexpr (sizeof(T) == 4) {
        if (variant == 1) launch_chained(k_clover_parts<T, 4>, grid, 128, st, g, L, parts);
        else if (variant == 2) launch_chained(k_clover_parts<T, 5>, grid, 128, st, g, L, parts);
        else launch_chained(k_clover_parts<T, 6>, grid, 128, st, g, L, parts);
    } else {
        if (variant == 1) launch_chained(k_clover_parts<T, 3>, grid, 128, st, g, L, parts);
        else launch_chained(k_clover_parts<T, 4>, grid, 128, st, g, L, parts);
    }
}

template <typename T>
void launch_observables(const Geom &g, const LinkField<T> &L, const PlaneParts<T> &parts, const ObsPlan &plan,
                        double *partial, double *out, int variant, cudaStream_t st) {
    clover_parts(g, L, parts, variant, st);
    launch_chained(k_plane_combine<T, OBS_SUMS>, plan.nblocks, plan.B, st, g, parts, plan.nb, plan.Bv, partial,
                   static_cast<double *>(nullptr), static_cast<double *>(nullptr));
    launch_obs_finalize(g, plan.nb, 1, partial, out, st);
}
template <typename T>
void launch_observables_density(const Geom &g, const LinkField<T> &L, const PlaneParts<T> &parts, const ObsPlan &plan,
                                double *partial, double *out, double *dq, double *de, cudaStream_t st) {
    clover_parts(g, L, parts, 0, st);
    launch_chained(k_plane_combine<T, OBS_DENSITY>, plan.nblocks, plan.B, st, g, parts, plan.nb, plan.Bv, partial, dq, de);
    launch_obs_finalize(g, plan.nb, 1, partial, out, st);
}
template <typename T>
void launch_weinberg(const Geom &g, const LinkField<T> &L, const PlaneParts<T> &parts, const ObsPlan &plan,
                     double *partial4, double *out, cudaStream_t st) {
    clover_parts(g, L, parts, 0, st);
    launch_chained(k_plane_combine<T, OBS_WEINBERG>, plan.nblocks, plan.B, st, g, parts, plan.nb, plan.Bv, partial4,
                   static_cast<double *>(nullptr), static_cast<double *>(nullptr));
    launch_chained(k_weinberg_finalize, 1, 1024, st, g.N[3], plan.nb, g.V, partial4, out);
}

#define GLAC_OBS_INST(T)                                                                                             \
    template void launch_observables<T>(const Geom &, const LinkField<T> &, const PlaneParts<T> &, const ObsPlan &,   \
                                        double *, double *, int, cudaStream_t);                                       \
    template void launch_observables_density<T>(const Geom &, const LinkField<T> &, const PlaneParts<T> &,            \
                                                const ObsPlan &, double *, double *, double *, double *,              \
                                                cudaStream_t);                                                        \
    template void launch_weinberg<T>(const Geom &, const LinkField<T> &, const PlaneParts<T> &, const ObsPlan &,      \
                                     double *, double *, cudaStream_t);
GLAC_OBS_INST(double)
GLAC_OBS_INST(float)
#undef GLAC_OBS_INST

}  // namespace glac
