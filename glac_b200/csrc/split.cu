// Small lattices: the work of one link over three warps.
//
// Where a lattice has fewer links than the GPU has thread slots, a thread per
// link leaves a stage as long as one thread's own chain of loads and products.
// Here a block takes 32 links and gives each of a link's three planes a warp:
// both staple terms, the force part of their sum and, in a measured stage 0,
// the plane's clover parts; one warp adds the three force parts and updates the
// links.  The stages of a step are launched so that one may start while the one
// before it drains (each waits for its end before the first field load).
#include "kernels.cuh"
#include "flow_body.cuh"
#include "launch.cuh"

#include <stdexcept>

namespace glac {

constexpr int kSplitWarps = 3;

// Anti-Hermitian matrices of a block's 32 links in shared memory, 16-byte chunks with the lane fastest.
template <typename T> struct LaneSlots;
template <> struct LaneSlots<float> {
    float4 p[kSplitWarps][2][32];
    __device__ __forceinline__ AH8<float> load(int k, int lane) const {
        const float4 u = p[k][0][lane], v = p[k][1][lane];
        AH8<float> Z;
        Z.a = u.x; Z.d = u.y; Z.b = cx(u.z, u.w); Z.c = cx(v.x, v.y); Z.e = cx(v.z, v.w);
        return Z;
    }
    __device__ __forceinline__ void store(int k, int lane, const AH8<float> &Z) {
        p[k][0][lane] = make_float4(Z.a, Z.d, Z.b.re, Z.b.im);
        p[k][1][lane] = make_float4(Z.c.re, Z.c.im, Z.e.re, Z.e.im);
    }
};
template <> struct LaneSlots<double> {
    double2 p[kSplitWarps][4][32];
    __device__ __forceinline__ AH8<double> load(int k, int lane) const {
        const double2 u = p[k][0][lane], v = p[k][1][lane], w = p[k][2][lane], x = p[k][3][lane];
        AH8<double> Z;
        Z.a = u.x; Z.d = u.y; Z.b = cx(v.x, v.y); Z.c = cx(w.x, w.y); Z.e = cx(x.x, x.y);
        return Z;
    }
    __device__ __forceinline__ void store(int k, int lane, const AH8<double> &Z) {
        p[k][0][lane] = make_double2(Z.a, Z.d);
        p[k][1][lane] = make_double2(Z.b.re, Z.b.im);
        p[k][2][lane] = make_double2(Z.c.re, Z.c.im);
        p[k][3][lane] = make_double2(Z.e.re, Z.e.im);
    }
};

// MEAS (stage 0): the clover parts of the input field, as k_flow_stage0_meas.
// COMBINE (stage 1): the blocks of direction 0 also combine the parts of their
// 32 sites into the partial sums of a 32-site plan.
// Eight (FP32) and five (FP64) blocks of three warps per SM; FP64's measured stage 0,
// which spills 180 B so, four: 31.0 us per measured step of 8^3 x 16 on B200, not 32.9.
template <typename T, int STAGE, bool MEAS, bool COMBINE>
__global__ void __launch_bounds__(32 * kSplitWarps, sizeof(T) == 4 ? 8 : MEAS ? 4 : 5)
    k_flow_split(Geom g, LinkField<T> in, LinkField<T> out, ForceField<T> zf, T alpha, T beta, CloverParts<T> cp,
                 double *partial) {
    __shared__ LaneSlots<T> slot;
    __shared__ T plq[kSplitWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int plane = blockIdx.x & 7, mu = plane >> 1, p = plane & 1, q = p ^ 1;
    const int s0 = (blockIdx.x >> 3) * 32;
    const bool valid = s0 + lane < g.Vh;
    const int s = valid ? s0 + lane : g.Vh - 1;
    const Site n = site_from_ps(g, p, s);
    const int nu = w + (w >= mu ? 1 : 0);
    const int f_mu = step_offset(g, n, mu, +1), b_nu = step_offset(g, n, nu, -1);
    const int s_mu = (n.lex + f_mu) >> 1, s_nup = (n.lex + step_offset(g, n, nu, +1)) >> 1;
    const int s_num = (n.lex + b_nu) >> 1, s_diag = (n.lex + f_mu + b_nu) >> 1;
    chain_wait();
    {
        // full products in FP32 too: three of them are short beside the loads, and
        // the clover keeps the accuracy of the stand-alone measurement
        M3<T> A = mul_nd(mul_nd(in.load(nu, q, s_mu), in.load(mu, q, s_nup)), in.load(nu, p, s));
        const M3<T> S = mul(mul_dd(in.load(nu, p, s_diag), in.load(mu, q, s_num)), in.load(nu, q, s_num));
        const M3<T> U = in.load(mu, p, s);
        if (MEAS) {
            T plaq = T(0);
            if (meas_takes(mu, nu)) {
                M3<T> W = A;
                plaq = retr_mul(U, W);
                sub_from(W, S);
                const bool neg = nu < mu;
                const int pl = neg ? plane_of(nu, mu) : plane_of(mu, nu);
                if (valid) {
                    cp.ah.store(2 * pl, p, s, clover_part(U, W, neg));
                    cp.ah.store(2 * pl + 1, q, s_mu, clover_part(W, U, neg));
                }
            }
            plq[w][lane] = plaq;
        }
        add_to(A, S);
        slot.store(w, lane, flow_force(U, A));
    }
    __syncthreads();
    if (w == 0) {
        const AH8<T> Z = ah_add(ah_add(slot.load(0, lane), slot.load(1, lane)), slot.load(2, lane));
        if (valid) flow_update<T, EXP_MORNINGSTAR, STAGE>(in.load(mu, p, s), Z, out, zf, alpha, beta, mu, p, s);
    } else if (MEAS && w == 1) {
        if (valid) cp.plaq[(mu * 2 + p) * g.Vh + s] = plq[0][lane] + plq[1][lane] + plq[2][lane];
    } else if (COMBINE && w == 1 && mu == 0) {
        const int half_slice = g.Vh / g.N[3], nb = half_slice >> 5;
        const int t = s0 / half_slice, j = (s0 - t * half_slice) >> 5;
        double plaq = 0.0, en = 0.0, qt = 0.0;
        combine_site(g, cp, p, s, plaq, en, qt);
        plaq = warp_sum_d(plaq);
        en = warp_sum_d(en);
        qt = warp_sum_d(qt);
        if (lane == 0) {
            double *o = partial + 3 * ((t * 2 + p) * nb + j);
            o[0] = plaq; o[1] = en; o[2] = qt;
        }
    }
}

bool flow_split_combines(const Geom &g) { return (g.Vh / g.N[3]) % 32 == 0; }

template <typename T>
void launch_flow_split(const Geom &g, const LinkField<T> &in, const LinkField<T> &out, const ForceField<T> &zf,
                       int stage, double alpha, double beta, const CloverParts<T> *meas, double *partial,
                       cudaStream_t st) {
    const CloverParts<T> cp = meas ? *meas : CloverParts<T>();
    auto kernel = stage == 0   ? (meas ? k_flow_split<T, 0, true, false> : k_flow_split<T, 0, false, false>)
                  : stage == 1 ? (meas ? k_flow_split<T, 1, false, true> : k_flow_split<T, 1, false, false>)
                               : k_flow_split<T, 2, false, false>;
    launch_chained(kernel, 8 * ((g.Vh + 31) / 32), 32 * kSplitWarps, st, g, in, out, zf, (T)alpha, (T)beta, cp, partial);
}
template void launch_flow_split<double>(const Geom &, const LinkField<double> &, const LinkField<double> &,
                                        const ForceField<double> &, int, double, double, const CloverParts<double> *,
                                        double *, cudaStream_t);
template void launch_flow_split<float>(const Geom &, const LinkField<float> &, const LinkField<float> &,
                                       const ForceField<float> &, int, double, double, const CloverParts<float> *,
                                       double *, cudaStream_t);

}  // namespace glac
