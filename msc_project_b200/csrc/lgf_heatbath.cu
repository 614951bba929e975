// Gauge-configuration generation on the GPU: hot/cold start, Cabibbo-Marinari
// heatbath with overrelaxation, and the average plaquette.
//
// Follows SU3_Heatbath (LGF/SU3_Heatbath/SU3_Heatbath.cpp): update(n) =
// n x (one heatbath sweep + OR_per_HB overrelaxation sweeps) (:16-25); a sweep
// visits the links by site parity and direction (:68-70, :117-119) and updates
// the three SU(2) subgroups (m,n) = (0,1), (0,2), (1,2) of each link in turn
// (:71-75), recomputing W = U * staple after every subgroup.  The SU(2)
// heatbath samples x0 by the reference's rejection scheme (:199-205), the
// overrelaxation reflects the subgroup (:78-104).
//
// B200 mapping: one launch per (parity, direction) class updates all its links
// in place in parallel, for more than a sweep or two on a copy of the links in
// parity order -- the staple of a link reads only other directions and
// opposite-parity links of its own direction, so the class has no internal
// dependencies.  Measured per class launch, FP64, against site order (same
// bits): 32x16^3 heatbath 40 -> 30 us, overrelaxation 33 -> 22; 24^3x48 197 ->
// 145 and 169 -> 109; FP32 105 -> 100 and 68 -> 60 on 24^3x48.
//  Random numbers come from a counter hash of (seed, class epoch,
// subgroup, site, draw), so results do not depend on the launch shape.  The
// rejection loop is bounded (HB_MAX_ATTEMPTS); a subgroup whose draws all
// fail is left unchanged and counted.  The reference seeds from
// std::random_device, so runs are compared statistically (average plaquette),
// not bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "lgf_engine.cuh"

namespace lgf {
namespace {

constexpr int HB_MAX_ATTEMPTS = 128;
constexpr int HB_DRAW_BITS = 10;  // draws per (epoch, subgroup, site): <= 2 + 4 * HB_MAX_ATTEMPTS < 1024

__device__ __forceinline__ double hb_draw(unsigned long long seed, unsigned long long base, int k) {
    return unit_open(seed, base + (unsigned long long)k);
}

// Longer runs of sweeps work on a copy of the links in parity order: the V/2 even sites, then
// the odd ones, each in site order, in the same 32-site blocks.  A class
// updates and reads whole runs of one parity there, where in site order every
// second site of a run is of the other parity and half of each 32-byte sector
// that a warp fetches goes unused -- and L2 bandwidth is what bounds a class
// (32x16^3, FP64: 12 TB/s in site order).  The copy takes the ring's second
// buffer, free between flows.
//
// N3 is even, so each (x0, x1, x2) row holds h = N3/2 sites of each parity:
// site x of parity p is entry row * h + k of its parity, x3 = 2k + o with
// o = (p + x0 + x1 + x2) & 1.  A step along x0, x1 or x2 keeps k and o; a step
// along x3 flips o and moves k by one when it leaves the pair.
struct ParitySite {
    int x0, x1, x2;  // coordinates of the row
    int row, k, o, p;
};
__host__ __device__ __forceinline__ ParitySite parity_site(const Geom& g, int p, int t) {
    const int h = g.n[3] >> 1;
    ParitySite a;
    a.p = p;
    a.row = t / h;
    a.k = t - a.row * h;
    a.x2 = a.row % g.n[2];
    const int r1 = a.row / g.n[2];
    a.x1 = r1 % g.n[1];
    a.x0 = r1 / g.n[1];
    a.o = (p + a.x0 + a.x1 + a.x2) & 1;
    return a;
}
// entry of the parity-ordered links
__host__ __device__ __forceinline__ int parity_index(const Geom& g, const ParitySite& a) {
    return (a.p ? g.V >> 1 : 0) + a.row * (g.n[3] >> 1) + a.k;
}
__host__ __device__ __forceinline__ int site_index(const Geom& g, const ParitySite& a) { return a.row * g.n[3] + 2 * a.k + a.o; }
__host__ __device__ __forceinline__ ParitySite parity_step(const Geom& g, ParitySite a, int d, int sign) {
    a.p ^= 1;
    if (d == 3) {
        const int h = g.n[3] >> 1;
        if (sign > 0 && a.o == 1) a.k = a.k == h - 1 ? 0 : a.k + 1;
        if (sign < 0 && a.o == 0) a.k = a.k == 0 ? h - 1 : a.k - 1;
        a.o ^= 1;
        return a;
    }
    const int n = sel4(d, g.n[0], g.n[1], g.n[2], 0), x = sel4(d, a.x0, a.x1, a.x2, 0);
    const int rows = d == 0 ? g.n[1] * g.n[2] : (d == 1 ? g.n[2] : 1);
    const int move = sign > 0 ? (x == n - 1 ? 1 - n : 1) : (x == 0 ? n - 1 : -1);
    a.row += move * rows;
    if (d == 0) a.x0 += move;
    if (d == 1) a.x1 += move;
    if (d == 2) a.x2 += move;
    return a;
}

// links of site order -> parity order (TO) or back
template <typename R, bool TO>
__global__ void __launch_bounds__(128) k_parity_order(const cplx<R>* __restrict__ in, cplx<R>* __restrict__ out, Geom g) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, mu = blockIdx.y;
    if (t >= g.V) return;
    const int half = g.V >> 1;
    const ParitySite a = parity_site(g, t >= half, t >= half ? t - half : t);
    const int s = site_index(g, a);
    store_link(out, g.V, mu, TO ? t : s, load_link(in, g.V, mu, TO ? s : t));
}

// the staple sum of staple_sum() (same products in the same order) on parity-ordered links
template <typename R>
__device__ __forceinline__ su3<R> staple_sum_parity(const cplx<R>* U, const Geom& g, const ParitySite& x, int mu) {
    const int V = g.V;
    su3<R> S;
    su3_zero(S);
    const int s = parity_index(g, x), xpm = parity_index(g, parity_step(g, x, mu, 1));
#pragma unroll
    for (int nu = 0; nu < 4; ++nu) {
        if (nu == mu) continue;
        const ParitySite m = parity_step(g, x, nu, -1);
        const int xpn = parity_index(g, parity_step(g, x, nu, 1)), xmn = parity_index(g, m);
        const int xmnpm = parity_index(g, parity_step(g, m, mu, 1));
        {
            const su3<R> t = mul_nn_su3(load_link(U, V, nu, s), load_link(U, V, mu, xpn));
            acc_na(S, load_link(U, V, nu, xpm), t);
        }
        {
            const su3<R> t = mul_nn_su3(load_link(U, V, mu, xmn), load_link(U, V, nu, xmnpm));
            acc_an(S, t, load_link(U, V, nu, xmn));
        }
    }
    return S;
}

// One (parity, direction) class of links in parity order, or (PARITY false) in
// site order; the same bits either way.  MINB: resident blocks per SM that the
// registers are capped for (heatbath_kernel).
template <typename R, int MINB, bool PARITY>
__global__ void __launch_bounds__(128, MINB) k_checkerboard(cplx<R>* U, Geom g, int mu, int parity, double beta,
                                                            unsigned long long seed, unsigned long long epoch, int overrelax,
                                                            unsigned int* __restrict__ failures) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (g.V >> 1)) return;
    const ParitySite x = parity_site(g, parity, t);
    const int s = site_index(g, x), at = PARITY ? parity_index(g, x) : s;  // the random numbers are keyed by the site
    su3<R> A;
    if constexpr (PARITY) A = staple_sum_parity<R>(U, g, x, mu);
    else A = staple_sum<R>(U, g, s, site_coord(g, s), mu);
    su3<R> u = load_link(U, g.V, mu, at);
#pragma unroll 1
    for (int sg = 0; sg < 3; ++sg) {
        const int m = sg == 2 ? 1 : 0, n = sg == 0 ? 1 : 2;  // (0,1), (0,2), (1,2)
        // the 2x2 block of W = u * A on rows/columns (m, n)
        cplx<double> w[2][2];
        const int rc[2] = {m, n};
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                cplx<double> acc = cmk<double>(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const cplx<R> x = u.m[3 * rc[a] + k], y = A.m[3 * k + rc[b]];
                    acc = cfma(cmk<double>(x.re, x.im), cmk<double>(y.re, y.im), acc);
                }
                w[a][b] = acc;
            }
        // O(4) coordinates of the subgroup block (GetSU2submatrix_O4_rep, SU3_mat.cpp:456-465)
        double r[4] = {w[0][0].re + w[1][1].re, w[0][1].im + w[1][0].im, w[0][1].re - w[1][0].re,
                       w[0][0].im - w[1][1].im};
        cplx<double> T[4];
        bool apply = true;
        if (overrelax) {  // SU3_Heatbath.cpp:78-99
            const double a = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3]);
            double q[4] = {1.0, 0.0, 0.0, 0.0};
            if (a >= 0.00001) {
                const double ia = 1.0 / a;
                q[0] = ia * r[0];
                q[1] = -ia * r[1];
                q[2] = -ia * r[2];
                q[3] = -ia * r[3];
            }
            const double z0 = q[0] * q[0] - q[1] * q[1] - q[2] * q[2] - q[3] * q[3];
            const double z1 = 2.0 * q[0] * q[1], z2 = 2.0 * q[0] * q[2], z3 = 2.0 * q[0] * q[3];
            T[0] = cmk<double>(z0, z3);
            T[1] = cmk<double>(z2, z1);
            T[2] = cmk<double>(-z2, z1);
            T[3] = cmk<double>(z0, -z3);
        } else {  // SU3_Heatbath.cpp:169-223
            const double norm = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3]);
            const double alpha = norm * beta / 3.0;
            const double in = 1.0 / norm;
            const cplx<double> sub[4] = {cmk<double>(r[0] * in, -r[3] * in), cmk<double>(-r[2] * in, -r[1] * in),
                                         cmk<double>(r[2] * in, -r[1] * in), cmk<double>(r[0] * in, r[3] * in)};
            const unsigned long long base =
                ((((epoch * 3ull + (unsigned long long)sg) * (unsigned long long)g.V) + (unsigned long long)s)
                 << HB_DRAW_BITS);
            const double two_pi = 6.28318530717958647692;
            double delta = 0.0;
            bool ok = false;
            int k = 0;
            for (int it = 0; it < HB_MAX_ATTEMPTS && !ok; ++it) {
                const double X = -log(1.0 - hb_draw(seed, base, k++));
                const double Xp = -log(1.0 - hb_draw(seed, base, k++));
                const double cc = cos(two_pi * hb_draw(seed, base, k++));
                delta = (Xp + X * cc * cc) / alpha;
                const double u4 = hb_draw(seed, base, k++);
                ok = u4 * u4 <= 1.0 - 0.5 * delta;
            }
            if (!ok) {
                atomicAdd(failures, 1u);
                apply = false;
            } else {
                const double x0 = 1.0 - delta;
                const double ax = sqrt(fmax(0.0, 1.0 - x0 * x0));
                const double ct = 2.0 * hb_draw(seed, base, k++) - 1.0;
                const double phi = two_pi * hb_draw(seed, base, k++);
                const double st = sqrt(fmax(0.0, 1.0 - ct * ct));
                double sp, cp;
                sincos(phi, &sp, &cp);
                const double x1 = ax * st * cp, x2 = ax * st * sp, x3 = ax * ct;
                const cplx<double> Vm[4] = {cmk<double>(x0, x3), cmk<double>(x2, x1), cmk<double>(-x2, x1),
                                            cmk<double>(x0, -x3)};
                T[0] = cadd(cmul(Vm[0], sub[0]), cmul(Vm[1], sub[2]));
                T[1] = cadd(cmul(Vm[0], sub[1]), cmul(Vm[1], sub[3]));
                T[2] = cadd(cmul(Vm[2], sub[0]), cmul(Vm[3], sub[2]));
                T[3] = cadd(cmul(Vm[2], sub[1]), cmul(Vm[3], sub[3]));
            }
        }
        if (apply) {  // rows m, n of u <- T * (rows m, n)   (SU3_Heatbath.cpp:100-104, 131-135)
#pragma unroll
            for (int col = 0; col < 3; ++col) {
                const cplx<double> um = cmk<double>(u.m[3 * m + col].re, u.m[3 * m + col].im);
                const cplx<double> un = cmk<double>(u.m[3 * n + col].re, u.m[3 * n + col].im);
                const cplx<double> nm = cadd(cmul(T[0], um), cmul(T[1], un));
                const cplx<double> nn = cadd(cmul(T[2], um), cmul(T[3], un));
                u.m[3 * m + col] = cmk<R>((R)nm.re, (R)nm.im);
                u.m[3 * n + col] = cmk<R>((R)nn.re, (R)nn.im);
            }
        }
    }
    store_link(U, g.V, mu, at, u);
}

// Random SU(3) per link as a product of three random SU(2) subgroup elements
// (Random::rnd_SU3_Group_elem, LGF/Math/Random.h:37-64): InitializeHotStart.
template <typename R>
__global__ void k_hot_start(cplx<R>* __restrict__ U, int V, unsigned long long seed) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * V) return;
    const int mu = t / V, s = t - mu * V;
    const unsigned long long base = ((unsigned long long)s * 4ull + (unsigned long long)mu) * 16ull;
    const double PI = 3.14159265358979323846;
    su3<double> out;
    su3_zero(out);
    out.m[0] = out.m[4] = out.m[8] = cmk<double>(1.0, 0.0);
    int k = 0;
    const int I[3] = {0, 0, 1}, J[3] = {1, 2, 2};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int i = I[q], j = J[q];
        const double alpha = PI * unit_open(seed, base + k++);
        const double phi = 2.0 * PI * unit_open(seed, base + k++);
        const double ct = 2.0 * unit_open(seed, base + k++) - 1.0;
        const double st = sqrt(1.0 - ct * ct);
        double sa, ca, sp, cp;
        sincos(alpha, &sa, &ca);
        sincos(phi, &sp, &cp);
        const double a0 = ca, a1 = sa * cp * st, a2 = sa * sp * st, a3 = sa * ct;
        su3<double> tmp;
        su3_zero(tmp);
        tmp.m[0] = tmp.m[4] = tmp.m[8] = cmk<double>(1.0, 0.0);
        tmp.m[3 * i + i] = cmk<double>(a0, a3);
        tmp.m[3 * i + j] = cmk<double>(a2, a1);
        tmp.m[3 * j + i] = cmk<double>(-a2, a1);
        tmp.m[3 * j + j] = cmk<double>(a0, -a3);
        out = mul_nn(tmp, out);
    }
    su3<R> o;
#pragma unroll
    for (int q = 0; q < 9; ++q) o.m[q] = cmk<R>((R)out.m[q].re, (R)out.m[q].im);
    store_link(U, V, mu, s, o);
}

template <typename R>
__global__ void k_cold_start(cplx<R>* __restrict__ U, int V) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * V) return;
    const int mu = t / V, s = t - mu * V;
    su3<R> o;
    su3_zero(o);
    o.m[0] = o.m[4] = o.m[8] = cmk<R>(R(1), R(0));
    store_link(U, V, mu, s, o);
}

// per block: sum over its sites of sum_{mu<nu} ReTr P_mu_nu(x)
template <typename R>
__global__ void __launch_bounds__(256) k_plaquette(const cplx<R>* __restrict__ U, Geom g, double* __restrict__ partial) {
    __shared__ double sh[256];
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    double acc = 0.0;
    if (s < g.V) {
        const Coord c = site_coord(g, s);
#pragma unroll
        for (int mu = 0; mu < 4; ++mu)
#pragma unroll
            for (int nu = mu + 1; nu < 4; ++nu) {
                const su3<R> a = load_link(U, g.V, mu, s);
                const su3<R> b = load_link(U, g.V, nu, fwd(g, s, mu, c.x[mu]));
                const su3<R> cc = load_link(U, g.V, mu, fwd(g, s, nu, c.x[nu]));
                const su3<R> d = load_link(U, g.V, nu, s);
                // ReTr U_mu(x) U_nu(x+mu) (U_nu(x) U_mu(x+nu))^dag: entry by entry, no third product
                const su3<R> ab = mul_nn(a, b);
                const su3<R> dc = mul_nn(d, cc);
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    R row = R(0);
#pragma unroll
                    for (int k = 3 * r; k < 3 * r + 3; ++k) row = fma(ab.m[k].re, dc.m[k].re, fma(ab.m[k].im, dc.m[k].im, row));
                    acc += (double)row;
                }
            }
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// The class kernel for nb blocks: of the register caps (blocks per SM) the one
// whose waves cost least, a full wave of m blocks per SM taken as cost[m].
// FP64: 3 blocks (168 registers) 1, 4 (128, some spills) 1.3: 32x16^3 runs one
// wave of 4 instead of two of 3, 22 against 24 us; 24^3x48 6 of 3, not 5 of 4.
// FP32: 4 blocks (128) 4 (4.2 in parity order), 5 (96) 5.05, 6 (80, some spills)
// 6.2 (6.9): many waves cost about the same with each cap, and 192000 sites fit
// one wave of 6 (overrelaxation of 4 sweeps in parity order 591 us, 674 in two
// waves of 5).  In parity order three waves of 6 lose to four of 5: 24^3x48, 4
// overrelaxation sweeps, 2205 against 2140 us.
template <typename R, bool PARITY> auto heatbath_kernel(int nb, int sms) {
    auto waves = [&](int per_sm) { return (nb + per_sm * sms - 1) / (per_sm * sms); };
    if constexpr (sizeof(R) == sizeof(double)) {
        return 10 * waves(3) > 13 * waves(4) ? k_checkerboard<R, 4, PARITY> : k_checkerboard<R, 3, PARITY>;
    } else {
        const int c4 = (PARITY ? 420 : 400) * waves(4), c5 = 505 * waves(5), c6 = (PARITY ? 690 : 620) * waves(6);
        if (c6 < c4 && c6 < c5) return k_checkerboard<R, 6, PARITY>;
        return c5 < c4 ? k_checkerboard<R, 5, PARITY> : k_checkerboard<R, 4, PARITY>;
    }
}

// n_iter x (heatbath sweep unless or_only, then or_per_hb overrelaxation sweeps)
template <typename R>
int heatbath_impl(lgf_ctx* ctx, lgf_lattice* lat, double beta, int n_iter, int or_per_hb, unsigned long long seed,
                  unsigned long long* rejected, bool or_only) {
    LatticeBuf& b = lat->buf;
    unsigned int* dfail = reinterpret_cast<unsigned int*>(b.slot);  // (a flow resets its slot before it counts)
    LGF_CUDA_TRY(ctx, cudaMemsetAsync(dfail, 0, sizeof(unsigned int), ctx->stream));
    const int V = b.g.V, th = 128, nb = (V / 2 + th - 1) / th;
    // The copy to parity order and back costs about as much as it saves in one
    // FP64 sweep, or in FP32, where a heatbath class gains little, in two
    // overrelaxation sweeps; while L2 holds both copies and they are more than a
    // few blocks per SM, in less.  Parity against site order, us, each with its
    // best register cap: FP64 one heatbath sweep 24^3x48 1680 against 1470, one
    // overrelaxation sweep 1280 against 1190 (160000 to 331776 sites 3 to 5% the
    // other way), one of each 2460 against 2580; FP32 one of each 24^3x48 1455
    // against 1405, 16^4 267 against 250, but 32x16^3 344 against 360 and
    // 221184 sites 489 against 505; one and two overrelaxation sweeps more on
    // 24^3x48 1890 against 1900, four 2030 against 2140.
    const long long heat = or_only ? 0 : n_iter, over = (long long)n_iter * or_per_hb, sweeps = heat + over;
    const bool parity = sizeof(R) == sizeof(double) || (V > 80000 && V < 250000) ? sweeps >= 2 : sweeps >= 4 || heat + 2 * over >= 5;
    cplx<R>*U = (cplx<R>*)b.U[0], *P = parity ? (cplx<R>*)b.U[1] : U;
    const dim3 order((V + th - 1) / th, 4);
    cudaError_t e = cudaSuccess;
    const bool any = n_iter > 0 && (!or_only || or_per_hb > 0);
    if (any && parity) k_parity_order<R, true><<<order, th, 0, ctx->stream>>>(U, P, b.g);
    auto sweep_class = parity ? heatbath_kernel<R, true>(nb, ctx->sm_count) : heatbath_kernel<R, false>(nb, ctx->sm_count);
    for (int it = 0; it < n_iter && e == cudaSuccess; ++it) {
        for (int sweep = or_only ? 1 : 0; sweep <= or_per_hb && e == cudaSuccess; ++sweep) {
            const int over = sweep > 0;
            for (int par = 0; par <= 1; ++par)
                for (int mu = 0; mu < 4; ++mu) {
                    const unsigned long long epoch = lat->hb_epoch++;
                    sweep_class<<<nb, th, 0, ctx->stream>>>(P, b.g, mu, par, beta, seed, epoch, over, dfail);
                }
            e = cudaGetLastError();
        }
    }
    if (any && parity && e == cudaSuccess) {
        k_parity_order<R, false><<<order, th, 0, ctx->stream>>>(P, U, b.g);
        e = cudaGetLastError();
    }
    unsigned int h = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, dfail, sizeof h, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return set_error(ctx, LGF_ECUDA, "heatbath failed: %s", cudaGetErrorString(e));
    if (rejected) *rejected = h;
    return LGF_OK;
}

}  // namespace
}  // namespace lgf

using namespace lgf;

extern "C" {

int lgf_heatbath(lgf_lattice* lat, double beta, int n_iter, int or_per_hb, uint64_t seed, uint64_t* rejected) {
    if (!lat || n_iter < 0 || or_per_hb < 0 || !(beta > 0.0)) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    if ((long long)lat->buf.g.V * 3 * (long long)(lat->hb_epoch + 8LL * n_iter * (or_per_hb + 1)) >=
        (1LL << (63 - HB_DRAW_BITS)))
        return set_error(ctx, LGF_EINVAL, "heatbath random-number counter space exhausted for this lattice");
    unsigned long long rej = 0;
    const int rc = lat->buf.prec == LGF_PREC_FP64
                       ? heatbath_impl<double>(ctx, lat, beta, n_iter, or_per_hb, seed, &rej, false)
                       : heatbath_impl<float>(ctx, lat, beta, n_iter, or_per_hb, seed, &rej, false);
    if (rejected) *rejected = rej;
    return rc;
}

int lgf_overrelax(lgf_lattice* lat, int n_sweeps) {
    if (!lat || n_sweeps < 0) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    return lat->buf.prec == LGF_PREC_FP64 ? heatbath_impl<double>(ctx, lat, 1.0, 1, n_sweeps, 0, nullptr, true)
                                          : heatbath_impl<float>(ctx, lat, 1.0, 1, n_sweeps, 0, nullptr, true);
}

int lgf_hot_start(lgf_lattice* lat, uint64_t seed) {
    if (!lat) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    const int V = lat->buf.g.V, nb = (4 * V + 127) / 128;
    if (lat->buf.prec == LGF_PREC_FP64)
        k_hot_start<double><<<nb, 128, 0, ctx->stream>>>((cplx<double>*)lat->buf.U[0], V, seed);
    else
        k_hot_start<float><<<nb, 128, 0, ctx->stream>>>((cplx<float>*)lat->buf.U[0], V, seed);
    LGF_CUDA_TRY(ctx, cudaGetLastError());
    LGF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return LGF_OK;
}

int lgf_cold_start(lgf_lattice* lat) {
    if (!lat) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    const int V = lat->buf.g.V, nb = (4 * V + 127) / 128;
    if (lat->buf.prec == LGF_PREC_FP64)
        k_cold_start<double><<<nb, 128, 0, ctx->stream>>>((cplx<double>*)lat->buf.U[0], V);
    else
        k_cold_start<float><<<nb, 128, 0, ctx->stream>>>((cplx<float>*)lat->buf.U[0], V);
    LGF_CUDA_TRY(ctx, cudaGetLastError());
    LGF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return LGF_OK;
}

int lgf_plaquette(lgf_lattice* lat, double* avg) {
    if (!lat || !avg) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    const Geom g = lat->buf.g;
    const int nb = (g.V + 255) / 256;
    double* dp = (double*)lat->buf.U[1];  // the ring's second buffer, free between flows
    if (lat->buf.prec == LGF_PREC_FP64)
        k_plaquette<double><<<nb, 256, 0, ctx->stream>>>((const cplx<double>*)lat->buf.U[0], g, dp);
    else
        k_plaquette<float><<<nb, 256, 0, ctx->stream>>>((const cplx<float>*)lat->buf.U[0], g, dp);
    std::vector<double> h(nb);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), dp, sizeof(double) * nb, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return set_error(ctx, LGF_ECUDA, "plaquette failed: %s", cudaGetErrorString(e));
    double sum = 0.0;
    for (double v : h) sum += v;
    *avg = sum / (3.0 * 6.0 * (double)g.V);  // SU3_field::Avg_Plaquette (SU3_field.cpp:485-499)
    return LGF_OK;
}

}  // extern "C"
