// Metropolis on small lattices: the work of one link over eight warps.
//
// A thread per link takes 18 link loads, 12 products and then its hits one after
// another, 10 us a sub-sweep on B200 however few links there are.  Only the
// accept decisions have to follow one another.  Here a block takes 32 links: six
// warps load the staple's terms and form their first products, three add the
// staple up (a row each), all draw the hits' proposals, one walks through the hits
// with W = U A, and three apply what it accepted to U (a column each).  Every
// number comes from the same operations in the same order as in the one-thread
// kernel, so the chain is the same bit for bit.
#include "launch.cuh"
#include "metropolis.cuh"

namespace glac {

constexpr int kMetroWarps = 8, kHitBatch = 10;

// Matrices of 32 lanes in shared memory as 16-byte chunks, the lane fastest.
template <typename T> struct Chunk;
template <> struct Chunk<float> { typedef float4 type; static constexpr int n = 5; };     // 18 reals, one more, a spare
template <> struct Chunk<double> { typedef double2 type; static constexpr int n = 10; };
template <typename T> struct LaneMatrix { typename Chunk<T>::type p[Chunk<T>::n][32]; };

__device__ __forceinline__ void put(LaneMatrix<float> &m, int lane, const M3<float> &X, float r) {
#pragma unroll
    for (int k = 0; k < 4; k++)
        m.p[k][lane] = make_float4(X.e[2 * k].re, X.e[2 * k].im, X.e[2 * k + 1].re, X.e[2 * k + 1].im);
    m.p[4][lane] = make_float4(X.e[8].re, X.e[8].im, r, 0.f);
}
__device__ __forceinline__ void put(LaneMatrix<double> &m, int lane, const M3<double> &X, double r) {
#pragma unroll
    for (int k = 0; k < 9; k++) m.p[k][lane] = make_double2(X.e[k].re, X.e[k].im);
    m.p[9][lane] = make_double2(r, 0.0);
}
__device__ __forceinline__ M3<float> get(const LaneMatrix<float> &m, int lane, float &r) {
    M3<float> X;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float4 v = m.p[k][lane];
        X.e[2 * k] = cx(v.x, v.y);
        X.e[2 * k + 1] = cx(v.z, v.w);
    }
    const float4 v = m.p[4][lane];
    X.e[8] = cx(v.x, v.y);
    r = v.z;
    return X;
}
__device__ __forceinline__ M3<double> get(const LaneMatrix<double> &m, int lane, double &r) {
    M3<double> X;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const double2 v = m.p[k][lane];
        X.e[k] = cx(v.x, v.y);
    }
    r = m.p[9][lane].x;
    return X;
}
// one element e < 9
__device__ __forceinline__ Cx<float> at(const LaneMatrix<float> &m, int lane, int e) {
    const float2 v = reinterpret_cast<const float2 *>(&m.p[e >> 1][lane])[e & 1];
    return cx(v.x, v.y);
}
__device__ __forceinline__ Cx<double> at(const LaneMatrix<double> &m, int lane, int e) {
    const double2 v = m.p[e][lane];
    return cx(v.x, v.y);
}
__device__ __forceinline__ void set(LaneMatrix<float> &m, int lane, int e, Cx<float> z) {
    reinterpret_cast<float2 *>(&m.p[e >> 1][lane])[e & 1] = make_float2(z.re, z.im);
}
__device__ __forceinline__ void set(LaneMatrix<double> &m, int lane, int e, Cx<double> z) {
    m.p[e][lane] = make_double2(z.re, z.im);
}

template <typename T> struct MetroShared {
    LaneMatrix<T> t[6];           // first products of the staple's terms
    LaneMatrix<T> A;              // the staple
    LaneMatrix<T> X[kHitBatch];   // proposals, each with its accept uniform
    uint32_t accepted[32];        // bit h: hit h of the batch
    float eps[32];                // learned spreads
    uint32_t feat[128];
};

template <typename T, bool LEARNED>
__global__ void __launch_bounds__(32 * kMetroWarps, sizeof(T) == 4 ? 3 : 2)
    k_metropolis_split(Geom g, LinkField<T> L, int mu, int p, T mfac, T eps, T sq1me, int nhits, uint32_t k0,
                       uint32_t k1, uint32_t sweep, uint32_t stream_id, unsigned long long *acc, Proposal P,
                       float beta) {
    extern __shared__ __align__(16) unsigned char smem[];
    MetroShared<T> &sh = *reinterpret_cast<MetroShared<T> *>(smem);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, q = p ^ 1;
    const bool valid = blockIdx.x * 32 + lane < g.Vh;
    const int s = valid ? blockIdx.x * 32 + lane : g.Vh - 1;
    const Site n = site_from_ps(g, p, s);
    const uint32_t link_id = (uint32_t)mu * (uint32_t)g.V + (uint32_t)n.lex;
    const int f_mu = step_offset(g, n, mu, +1), s_mu = (n.lex + f_mu) >> 1;
    auto direction = [&](int j) { return j + (j >= mu ? 1 : 0); };
    // warp 6 draws first, warps that form a term take fewer hits
    auto draw = [&](int h0, int count, T e, T sq) {
        for (int h = (w + 2) & (kMetroWarps - 1); h < count; h += kMetroWarps) {
            M3<T> X;
            T r;
            draw_proposal<T>(k0, k1, link_id, sweep, stream_id, h0 + h, e, sq, P.flips, X, r);
            put(sh.X[h], lane, X, r);
        }
    };
    chain_wait();
    if (w < 6) {
        const int nu = direction(w >> 1);
        M3<T> t;
        if (w & 1) {
            const int b_nu = step_offset(g, n, nu, -1), s_num = (n.lex + b_nu) >> 1;
            t = mul_dd(L.load(nu, p, (n.lex + f_mu + b_nu) >> 1), L.load(mu, q, s_num));
        } else {
            t = mul_nd(L.load(nu, q, s_mu), L.load(mu, q, (n.lex + step_offset(g, n, nu, +1)) >> 1));
        }
        put(sh.t[w], lane, t, T(0));
    }
    if (!LEARNED) draw(0, min(nhits, kHitBatch), eps, sq1me);
    __syncthreads();
    if (w < 3) {  // row w of the staple, term by term as staple() adds them
        Cx<T> a[3];
#pragma unroll
        for (int j = 0; j < 3; j++) a[j] = cx(T(0), T(0));
#pragma unroll 1
        for (int k = 0; k < 6; k++) {
            const int nu = direction(k >> 1);
            const Cx<T> t0 = at(sh.t[k], lane, 3 * w), t1 = at(sh.t[k], lane, 3 * w + 1),
                        t2 = at(sh.t[k], lane, 3 * w + 2);
            const bool low = k & 1;
            const M3<T> c = L.load(nu, low ? q : p, low ? (n.lex + step_offset(g, n, nu, -1)) >> 1 : s);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                if (low) {
                    a[j] = cmac(a[j], t0, c(0, j));
                    a[j] = cmac(a[j], t1, c(1, j));
                    a[j] = cmac(a[j], t2, c(2, j));
                } else {
                    a[j] = cmac_bc(a[j], t0, c(j, 0));
                    a[j] = cmac_bc(a[j], t1, c(j, 1));
                    a[j] = cmac_bc(a[j], t2, c(j, 2));
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 3; j++) set(sh.A, lane, 3 * w + j, a[j]);
    }
    __syncthreads();
    if (LEARNED) {
        if (w == 0) {
            T unused;
            float f[8];
            staple_features(get(sh.A, lane, unused), beta, f);
            sh.eps[lane] = mlp_spread_warp(f, P, sh.feat);
        }
        __syncthreads();
        eps = (T)sh.eps[lane];
        sq1me = sqrt(T(1) - eps * eps);
        draw(0, min(nhits, kHitBatch), eps, sq1me);
        __syncthreads();
    }
    M3<T> W;
    if (w == 0) {
        T unused;
        W = mul(L.load_rw(mu, p, s), get(sh.A, lane, unused));
    }
    // column w of U
    Cx<T> u[3];
    if (w < 3) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const auto v = *L.element(mu, p, s, 3 * i + w);
            u[i] = cx(v.x, v.y);
        }
    }
    uint32_t changed = 0;
    unsigned long long na = 0;
    for (int h0 = 0; h0 < nhits; h0 += kHitBatch) {
        const int count = min(nhits - h0, kHitBatch);
        if (h0 > 0) {
            __syncthreads();
            draw(h0, count, eps, sq1me);
            __syncthreads();
        }
        if (w == 0) {
            uint32_t bits = 0;
#pragma unroll 1
            for (int h = 0; h < count; h++) {
                T r;
                const M3<T> X = get(sh.X[h], lane, r);
                const T dS = (retr_mul(X, W) - retr(W)) * mfac;
                if (accept_weight<T>(dS) > r) {
                    W = mul(X, W);
                    bits |= 1u << h;
                }
            }
            if (!valid) bits = 0;
            na += __popc(bits);
            sh.accepted[lane] = bits;
        }
        __syncthreads();
        if (w < 3) {
            const uint32_t bits = sh.accepted[lane];
            changed |= bits;
#pragma unroll 1
            for (int h = 0; h < count; h++) {
                if (!(bits >> h & 1)) continue;
                T r;
                const M3<T> X = get(sh.X[h], lane, r);
                Cx<T> v[3];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    v[i] = X(i, 0) * u[0];
                    v[i] = cmac(v[i], X(i, 1), u[1]);
                    v[i] = cmac(v[i], X(i, 2), u[2]);
                }
#pragma unroll
                for (int i = 0; i < 3; i++) u[i] = v[i];
            }
        }
    }
    chain_release();
    if (w < 3 && changed) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
            auto *e = L.element(mu, p, s, 3 * i + w);
            e->x = u[i].re;
            e->y = u[i].im;
        }
    }
    if (w == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) na += __shfl_down_sync(0xffffffffu, na, o);
        if (lane == 0 && na) atomicAdd(acc, na);
    }
}

// Up to two blocks per SM, all of them resident; with a third the eight warps of a
// block, of which one walks the hits, cost more than they shorten.  Microseconds
// per sweep on B200, so / a thread per link: 8^3 x 16 FP32 65 / 84 (learned 83 / 100),
// FP64 87 / 123; 8^2 x 16^2 FP32 77 / 84, FP64 104 / 125; 10^3 x 20 (313 blocks) FP32
// 84 / 85, FP64 173 / 129.
bool metropolis_splits(const Geom &g) { return (g.Vh + 31) / 32 <= 2 * 148; }

template <typename T>
void launch_metropolis_split(const Geom &g, const LinkField<T> &L, int mu, int p, T mfac, T eps, T sq1me, int nhits,
                             uint32_t k0, uint32_t k1, uint32_t sweep, uint32_t stream_id, unsigned long long *acc,
                             const Proposal &P, float beta, cudaStream_t st) {
    auto kernel = P.net ? k_metropolis_split<T, true> : k_metropolis_split<T, false>;
    const int bytes = (int)sizeof(MetroShared<T>);
    // per device (cheap): the attribute is not shared between devices
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    launch_chained_shared(kernel, (unsigned)((g.Vh + 31) / 32), 32 * kMetroWarps, bytes, st, g, L, mu, p, mfac, eps, sq1me,
                          nhits, k0, k1, sweep, stream_id, acc, P, beta);
}
template void launch_metropolis_split<double>(const Geom &, const LinkField<double> &, int, int, double, double, double,
                                              int, uint32_t, uint32_t, uint32_t, uint32_t, unsigned long long *,
                                              const Proposal &, float, cudaStream_t);
template void launch_metropolis_split<float>(const Geom &, const LinkField<float> &, int, int, float, float, float, int,
                                             uint32_t, uint32_t, uint32_t, uint32_t, unsigned long long *,
                                             const Proposal &, float, cudaStream_t);

}  // namespace glac
