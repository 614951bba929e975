// sm_100a kernels of the Wilson-flow engine.
//
//   k_rk3_stage<R,S,PARTS>  one fused Luscher RK3 stage for every link (by size,
//                      stage_form: also k_rk3_split, or k_rk3_plaquettes +
//                      k_rk3_update): staple,
//                      projected force Z, su(3) accumulator update,
//                      Cayley-Hamilton exponential, link update (ping-pong).
//                      Replaces Wilson::calculate_FlowGradient
//                      (LGF/Action/Gauge/Wilson.cpp:55-71), SU3_field::staple
//                      (LGF/Field/SU3_field.cpp:519-530), HermTrLessExp
//                      (LGF/Math/SU3_mat.cpp:216-289) and the three update
//                      loops of GradientFlow::flow (GradientFlow.cpp:22-54).
//   k_measure<R>       small lattices: clover F (E) and improved F (q) for every
//                      site and plane in one launch, per-site e(x), q(x),
//                      warp-shuffle block partials by x0 slice (the others:
//                      lgf_measure.cuh).  Replaces EnergyDensity::calculate and
//                      TopologicalCharge::calculate (Observables/*.cpp) and the
//                      loop averages of SU3_field.cpp:533-792.
//   k_reduce           fixed-order FP64 reductions (per x0 slice, then global)
//                      in place of MPI_Allreduce; deterministic run to run.
//   k_to_device / k_to_file    file-order float64 <-> device layout
//   k_generate_G       synthetic links exp(i s sum_a h_a T^a)
//   k_reunitarize      FP32-mixed: Gram-Schmidt rows 0,1; row 2 = conj(r0 x r1)
//   k_unitarity        max ||U^dag U - 1||_F and |det U - 1| per block
//   k_debug_*          per-function outputs for parity tests
#pragma once
#include "lgf_lattice.cuh"

// Launch bounds of the RK3 stage: (max threads per block, min resident
// blocks per SM), which cap the registers per thread at 65536 / 384 = 170,
// i.e. 168 once rounded to the allocation unit.  double: 384-thread blocks
// (12 warps per SM: 7% faster per stage than 8 warps at 250 registers on
// 24^3x48 and 48^4); float: 128-thread blocks, three per SM (at 170
// registers the rounding to 176 leaves room for only two: 15% slower).
#ifndef LGF_STAGE_MAXT_D
#define LGF_STAGE_MAXT_D 384
#endif
#ifndef LGF_STAGE_MAXT_F
#define LGF_STAGE_MAXT_F 384
#endif
#ifndef LGF_STAGE_MINB
#define LGF_STAGE_MINB 1
#endif

namespace lgf {

// ----------------------------------------------------------------- staple
// Z = -1/2 [ (W - W^dag) - 1/3 Tr(W - W^dag) ],  W = U_mu(x) A,
// A = sum_{nu != mu} U_nu(x+mu) (U_nu(x) U_mu(x+nu))^dag
//                  + (U_mu(x-nu) U_nu(x-nu+mu))^dag U_nu(x-nu)
// S += the two staples of link (s, mu) in the plane of nu; xpm = s + mu, xn = the nu coordinate of s
template <typename R>
__device__ __forceinline__ void add_staples(su3<R>& S, const cplx<R>* __restrict__ U, const Geom& g, int s, int mu, const Dir& dm,
                                            int xpm, int nu, int xn) {
    const int V = g.V;
    const int xpn = fwd(g, s, nu, xn), xmn = bwd(g, s, nu, xn);
    const int xmnpm = fwd(xmn, dm);  // the mu coordinate of x-nu is x_mu
    {
        su3<R> a2 = load_link(U, V, nu, s);
        su3<R> a3 = load_link(U, V, mu, xpn);
        su3<R> t = mul_nn_su3(a2, a3);
        su3<R> a1 = load_link(U, V, nu, xpm);
        acc_na(S, a1, t);
    }
    {
        su3<R> b1 = load_link(U, V, mu, xmn);
        su3<R> b2 = load_link(U, V, nu, xmnpm);
        su3<R> t = mul_nn_su3(b1, b2);
        su3<R> b3 = load_link(U, V, nu, xmn);
        acc_an(S, t, b3);
    }
}

// PARTS: a sum per nu, added in order (the split form's grouping; in FP32 also
// 2 us per step faster than one sum up to 14208 sites)
template <typename R, bool PARTS = false>
__device__ __forceinline__ su3<R> staple_sum(const cplx<R>* __restrict__ U, const Geom& g, int s, const Coord& c, int mu) {
    const Dir dm = dir_of(g, c, mu);
    su3<R> S;
    su3_zero(S);
    const int xpm = fwd(s, dm);
    if (PARTS) {
#pragma unroll
        for (int part = 0; part < 3; ++part) {
            const int nu = part + (part >= mu ? 1 : 0);
            const int xn = sel4(nu, c.x[0], c.x[1], c.x[2], c.x[3]);
            if (part == 0) {
                add_staples(S, U, g, s, mu, dm, xpm, nu, xn);
            } else {
                su3<R> P;
                su3_zero(P);
                add_staples(P, U, g, s, mu, dm, xpm, nu, xn);
                su3_addto(S, P);
            }
        }
        return S;
    }
#pragma unroll
    for (int nu = 0; nu < 4; ++nu)
        if (nu != mu) add_staples(S, U, g, s, mu, dm, xpm, nu, c.x[nu]);
    return S;
}

// s times the traceless anti-Hermitian part of A B, W - W^dag - 1/3 Tr(W - W^dag),
// computing only what it reads of the product: the imaginary parts of the
// diagonal and the three off-diagonal pairs (90 real operations instead of 108)
template <typename R> __device__ __forceinline__ alg<R> ta_of_product(const su3<R>& A, const su3<R>& B, R s) {
    R d[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        R im = R(0);
#pragma unroll
        for (int k = 0; k < 3; ++k) im = fma(A.m[3 * i + k].re, B.m[3 * k + i].im, fma(A.m[3 * i + k].im, B.m[3 * k + i].re, im));
        d[i] = R(2) * im;
    }
    const R tr = (d[0] + d[1] + d[2]) * R(1.0 / 3.0);
    alg<R> z;
    z.v[0] = s * (d[0] - tr);
    z.v[1] = s * (d[1] - tr);
    const int I[3] = {0, 0, 1}, J[3] = {1, 2, 2};
#pragma unroll
    for (int o = 0; o < 3; ++o) {
        const int i = I[o], j = J[o];
        cplx<R> wij = cmul(A.m[3 * i], B.m[j]);
        wij = cfma(A.m[3 * i + 1], B.m[3 + j], wij);
        wij = cfma(A.m[3 * i + 2], B.m[6 + j], wij);
        cplx<R> wji = cmul(A.m[3 * j], B.m[i]);
        wji = cfma(A.m[3 * j + 1], B.m[3 + i], wji);
        wji = cfma(A.m[3 * j + 2], B.m[6 + i], wji);
        z.v[2 + 2 * o] = s * (wij.re - wji.re);
        z.v[3 + 2 * o] = s * (wij.im + wji.im);
    }
    return z;
}

template <typename R, bool PARTS = false>
__device__ __forceinline__ alg<R> flow_gradient(const cplx<R>* __restrict__ U, const Geom& g, int s, const Coord& c,
                                                int mu, su3<R>& u_out) {
    const su3<R> S = staple_sum<R, PARTS>(U, g, s, c, mu);
    u_out = load_link(U, g.V, mu, s);
    return ta_of_product(u_out, S, R(-0.5));
}

// Device descriptor of one resident lattice.  Every flow launch works on a
// table of these plus a work list of tiles, so one launch can cover one
// lattice or many lattices of uneven volumes (batch and serving forms).
template <typename R> struct LatDesc {
    Geom g;
    cplx<R>* U0;          // ring of link buffers: stage 1 U0->U1, 2 U1->U2, 3 U2->U0
    cplx<R>* U1;
    cplx<R>* U2;
    R* A;                 // su(3) RK3 accumulator, 8 coordinates per link
    double2* partial;     // [N0 * nchunk] block partials of the measurement
    double2* slice_sums;  // [N0]
    double* meas;         // [capacity * (2 + 2 N0)] measurement results
    int* slot;            // next measurement slot; slot[1]: slices summed so far (k_reduce)
    int nchunk;           // measurement blocks per x0 slice
    double eps;
};

// ---------------------------------------------------------- Wilson loops
// The clover-type averages of the reference (SU3_field.cpp:533-792) are sums
// of a x b rectangular loops through x, one per quadrant, in the orientation
//   q0: +nu^b +mu^a -nu^b -mu^a     q1: +mu^a -nu^b -mu^a +nu^b
//   q2: -mu^a +nu^b +mu^a -nu^b     q3: -nu^b -mu^a +nu^b +mu^a
// (a links along mu, b along nu).  With quadrant signs (sm, sn) = (+,+),
// (+,-), (-,+), (-,-), every leaf is  Pn Pm^dag  (q0, q3) or its adjoint
// (q1, q2), where Pn = (sn nu)^b (sm mu)^a and Pm = (sm mu)^a (sn nu)^b are
// the two L-shaped paths from x to the far corner.  The projection F[W] is
// linear and F[W^dag] = -F[W], so each quadrant adds sign * F[Pn Pm^dag]
// with sign = +1 for q0, q3 and -1 for q1, q2, weighted per shape:
//   F^ = 19/9 F[C11] + 1/36 F[C22] - 32/45 F[C12] + 1/15 F[C13]
//      C11 = 1/4 (1x1), C22 = 1/4 (2x2), C12 = 1/8 (1x2 + 2x1), C13 = 1/8 (1x3 + 3x1)
// (SU3_field.cpp:588-597), and the clover F = F[C11] for E.  The paths are
// built as shared chains (a path of a shape extends the path of the shape
// before it by one link) and from shared straight lines: 12 matrix products
// and 14 global link loads per quadrant (plane_fields_body) instead of 34 and
// 40 for separate loops.
struct PlanePos { int s, xm, xn; };

// A link of the device layout, or (FILE, double) of file-order links: entry k
// at (s * 4 + mu) * 9 + k.  There a lane's link is 144 contiguous bytes and
// the next lane's 576 further on, so a plain 16-byte load of a warp touches 32
// cache lines and takes the L1 as many cycles.  Two lanes therefore read their
// two links together, 32 contiguous bytes of one link at a time (16 lines per
// load), and exchange halves by a shuffle: every lane of the warp must call.
__device__ __forceinline__ cplx<double> shfl_xor_c(cplx<double> z, int mask) {
    return cmk<double>(__shfl_xor_sync(0xffffffffu, z.re, mask), __shfl_xor_sync(0xffffffffu, z.im, mask));
}
__device__ __forceinline__ cplx<double> pick(bool c, cplx<double> a, cplx<double> b) { return cmk<double>(c ? a.re : b.re, c ? a.im : b.im); }
template <bool FILE, typename R> __device__ __forceinline__ su3<R> load_link_from(const cplx<R>* __restrict__ U, int V, int mu, int s) {
    if constexpr (FILE) {
        static_assert(sizeof(R) == sizeof(double), "file-order links are double");
        const bool odd = threadIdx.x & 1;
        const int other = __shfl_xor_sync(0xffffffffu, s, 1);
        const cplx<R>* even_link = U + ((size_t)(odd ? other : s) * 4 + mu) * 9 + (odd ? 1 : 0);
        const cplx<R>* odd_link = U + ((size_t)(odd ? s : other) * 4 + mu) * 9 + (odd ? 1 : 0);
        su3<R> a;
#pragma unroll
        for (int k = 0; k < 8; k += 2) {  // this lane's entry (k, or k + 1 on odd lanes) of both links
            const cplx<R> e = ldc(even_link + k), o = ldc(odd_link + k);
            const cplx<R> r = shfl_xor_c(pick(odd, e, o), 1);
            a.m[k] = pick(odd, r, e);
            a.m[k + 1] = pick(odd, o, r);
        }
        a.m[8] = ldc(U + ((size_t)s * 4 + mu) * 9 + 8);
        return a;
    } else {
        return load_link(U, V, mu, s);
    }
}
// Links are read in R and multiplied in D; FILE: U is the caller's own array in
// file order instead of the device layout, and products are formed in full: the
// result is that of the matrices as given, also where they are not quite SU(3).
template <typename R, typename D = R, bool FILE = false> struct Plane {
    const cplx<R>* __restrict__ U;
    int V, mu, nu;
    Dir dm, dn;  // .x unused: positions carry their own coordinates

    // the link of one step from p and the new position; adjoint for a backward step
    __device__ __forceinline__ su3<D> step(PlanePos& p, bool along_mu, int sign) const {
        const Dir& d = along_mu ? dm : dn;
        int& xc = along_mu ? p.xm : p.xn;
        const int dir = along_mu ? mu : nu;
        if (sign > 0) {
            su3<D> l = su3_cast<D>(load_link_from<FILE>(U, V, dir, p.s));
            p.s = (xc == d.n - 1) ? p.s - (d.n - 1) * d.stride : p.s + d.stride;
            xc = wrap_inc(xc, d.n);
            return l;
        }
        p.s = (xc == 0) ? p.s + (d.n - 1) * d.stride : p.s - d.stride;
        xc = wrap_dec(xc, d.n);
        su3<D> l = su3_cast<D>(load_link_from<FILE>(U, V, dir, p.s));
        su3<D> a;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) a.m[3 * r + c] = cmk<D>(l.m[3 * c + r].re, -l.m[3 * c + r].im);
        return a;
    }
    // move p by count steps without loading links
    __host__ __device__ __forceinline__ void advance(PlanePos& p, bool along_mu, int sign, int count) const {
        const Dir& d = along_mu ? dm : dn;
        int& xc = along_mu ? p.xm : p.xn;
        for (int i = 0; i < count; ++i) {
            if (sign > 0) {
                p.s = (xc == d.n - 1) ? p.s - (d.n - 1) * d.stride : p.s + d.stride;
                xc = wrap_inc(xc, d.n);
            } else {
                p.s = (xc == 0) ? p.s + (d.n - 1) * d.stride : p.s - d.stride;
                xc = wrap_dec(xc, d.n);
            }
        }
    }
    // P <- P * (link of one step from p)
    __device__ __forceinline__ void ext(su3<D>& P, PlanePos& p, bool along_mu, int sign) const {
        const Dir& d = along_mu ? dm : dn;
        int& xc = along_mu ? p.xm : p.xn;
        const int dir = along_mu ? mu : nu;
        if (sign > 0) {
            const su3<D> l = su3_cast<D>(load_link_from<FILE>(U, V, dir, p.s));
            p.s = (xc == d.n - 1) ? p.s - (d.n - 1) * d.stride : p.s + d.stride;
            xc = wrap_inc(xc, d.n);
            P = FILE ? mul_nn(P, l) : mul_nn_su3(P, l);
        } else {
            p.s = (xc == 0) ? p.s + (d.n - 1) * d.stride : p.s - d.stride;
            xc = wrap_dec(xc, d.n);
            const su3<D> l = su3_cast<D>(load_link_from<FILE>(U, V, dir, p.s));
            P = FILE ? mul_na(P, l) : mul_na_su3(P, l);
        }
    }
};

// Where a measurement thread keeps its two 8-coordinate sums: registers, or
// (double, LGF_MEAS_SMEM_ACC) its own column of shared memory.  The FP64
// kernel holds two path matrices, the incoming link and these sums at its
// peak; at 168 registers that spilled ~0.6 KB per thread, and with the sums in
// shared memory (48 KB per block) it spills ~50 B and ran 12-13% faster when
// this kernel measured 16^4 to 48^4.  Same operations, same order, either way
// (bit-identical).
template <typename R> struct RegAcc {
    alg<R>& a;
    __device__ __forceinline__ R get(int k) const { return a.v[k]; }
    __device__ __forceinline__ void set(int k, R x) { a.v[k] = x; }
};
template <typename R> struct SmemAcc {
    R* p;  // coordinate k at p[k * MEAS_ACC_STRIDE]
    __device__ __forceinline__ R get(int k) const;
    __device__ __forceinline__ void set(int k, R x);
};

// F += c * F[A B^dag] without forming the product: only the entries the
// projection reads (Im of the diagonal, both triangles) are computed.
template <typename R, typename Acc> __device__ __forceinline__ void leaf_acc(const su3<R>& A, const su3<R>& B, R c, Acc F) {
    // W_ij = sum_k A_ik conj(B_jk)
    R d[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        R im = R(0);
#pragma unroll
        for (int k = 0; k < 3; ++k) im = fma(A.m[3 * i + k].im, B.m[3 * i + k].re, fma(-A.m[3 * i + k].re, B.m[3 * i + k].im, im));
        d[i] = im;
    }
    const R tr = (d[0] + d[1] + d[2]) * R(1.0 / 3.0);
    F.set(0, fma(c, d[0] - tr, F.get(0)));
    F.set(1, fma(c, d[1] - tr, F.get(1)));
    const int I[3] = {0, 0, 1}, J[3] = {1, 2, 2};
#pragma unroll
    for (int o = 0; o < 3; ++o) {
        const int i = I[o], j = J[o];
        cplx<R> wij = cmulc(A.m[3 * i], B.m[3 * j]);
        wij = cfmac(A.m[3 * i + 1], B.m[3 * j + 1], wij);
        wij = cfmac(A.m[3 * i + 2], B.m[3 * j + 2], wij);
        cplx<R> wji = cmulc(A.m[3 * j], B.m[3 * i]);
        wji = cfmac(A.m[3 * j + 1], B.m[3 * i + 1], wji);
        wji = cfmac(A.m[3 * j + 2], B.m[3 * i + 2], wji);
        // (-i/2)(a + ib) = (b/2, -a/2),  a + ib = W_ij - conj(W_ji)
        const R a = wij.re - wji.re, b = wij.im + wji.im;
        F.set(2 + 2 * o, fma(R(0.5) * c, b, F.get(2 + 2 * o)));
        F.set(3 + 2 * o, fma(R(-0.5) * c, a, F.get(3 + 2 * o)));
    }
}

__device__ __constant__ int c_plane_mu[6] = {0, 0, 0, 1, 1, 2};
__device__ __constant__ int c_plane_nu[6] = {1, 2, 3, 2, 3, 3};

// ---------------------------------------------------------------- fields
// Hermitian traceless field of 8 coordinates per site in 32-site blocks:
// double2 pairs or float4 quads, planes of 32 sites.
constexpr int FIELD_REALS = 8 * LAYOUT_BLOCK;  // one field of one block
template <typename R, bool RO> __device__ __forceinline__ alg<R> get_field(const R* p) {
    alg<R> z;
    if constexpr (sizeof(R) == sizeof(double)) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double2* a = reinterpret_cast<const double2*>(p) + q * LAYOUT_BLOCK;
            const double2 v = RO ? __ldg(a) : *a;
            z.v[2 * q] = v.x;
            z.v[2 * q + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float4* a = reinterpret_cast<const float4*>(p) + q * LAYOUT_BLOCK;
            const float4 v = RO ? __ldg(a) : *a;
            z.v[4 * q] = v.x;
            z.v[4 * q + 1] = v.y;
            z.v[4 * q + 2] = v.z;
            z.v[4 * q + 3] = v.w;
        }
    }
    return z;
}
template <typename R> __device__ __forceinline__ void put_field(R* p, const alg<R>& z) {
    if constexpr (sizeof(R) == sizeof(double)) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            reinterpret_cast<double2*>(p)[q * LAYOUT_BLOCK] = make_double2(z.v[2 * q], z.v[2 * q + 1]);
    } else {
#pragma unroll
        for (int q = 0; q < 2; ++q)
            reinterpret_cast<float4*>(p)[q * LAYOUT_BLOCK] = make_float4(z.v[4 * q], z.v[4 * q + 1], z.v[4 * q + 2], z.v[4 * q + 3]);
    }
}

// c F[A B^dag], computed in D and returned in R
template <typename R, typename D> __device__ __forceinline__ alg<R> leaf(const su3<D>& A, const su3<D>& B, D c) {
    alg<D> F;
#pragma unroll
    for (int k = 0; k < 8; ++k) F.v[k] = D(0);
    leaf_acc(A, B, c, RegAcc<D>{F});
    alg<R> z;
#pragma unroll
    for (int k = 0; k < 8; ++k) z.v[k] = (R)F.v[k];
    return z;
}

// U^dag H U of a Hermitian traceless H, in the same 8 coordinates: column by
// column, Y = H U_col (30 operations) and the entries of U^dag Y at and above
// the diagonal; the last diagonal entry follows from the trace.
template <typename R> __device__ __forceinline__ alg<R> shift(const alg<R>& h, const su3<R>& U) {
    const R a0 = h.v[0], a1 = h.v[1], a2 = -(h.v[0] + h.v[1]);
    const cplx<R> q01 = cmk<R>(h.v[2], h.v[3]), q02 = cmk<R>(h.v[4], h.v[5]), q12 = cmk<R>(h.v[6], h.v[7]);
    alg<R> z;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const cplx<R> u0 = U.m[c], u1 = U.m[3 + c], u2 = U.m[6 + c];
        const cplx<R> y0 = cfma(q02, u2, cfma(q01, u1, cmk<R>(a0 * u0.re, a0 * u0.im)));
        const cplx<R> y1 = cfma(q12, u2, ccfma(q01, u0, cmk<R>(a1 * u1.re, a1 * u1.im)));
        const cplx<R> y2 = ccfma(q12, u1, ccfma(q02, u0, cmk<R>(a2 * u2.re, a2 * u2.im)));
        if (c < 2) {
            R d = u0.re * y0.re;
            d = fma(u0.im, y0.im, d);
            d = fma(u1.re, y1.re, d);
            d = fma(u1.im, y1.im, d);
            d = fma(u2.re, y2.re, d);
            z.v[c] = fma(u2.im, y2.im, d);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (r >= c) continue;
            cplx<R> w = ccmul(U.m[r], y0);
            w = ccfma(U.m[3 + r], y1, w);
            w = ccfma(U.m[6 + r], y2, w);
            const int o = 2 * (r + c);  // 01 -> 2, 02 -> 4, 12 -> 6
            z.v[o] = w.re;
            z.v[o + 1] = w.im;
        }
    }
    return z;
}
template <typename R> __device__ __forceinline__ alg<R> alg_add(const alg<R>& x, const alg<R>& y) {
    alg<R> z;
#pragma unroll
    for (int k = 0; k < 8; ++k) z.v[k] = x.v[k] + y.v[k];
    return z;
}

// The tiles of one launch: seg->x .. + seg->y of the list, read on the device so
// that a captured graph follows the list; or, for a group that never changes
// (seg null), the range and its only member by value, which takes two of the
// four dependent loads (range, tile, descriptor, links) that open every kernel
// out of its latency: 1 to 1.5 us of an 8^4 step's three launches.
struct Work { const int2* seg; int first, count; };
__device__ __forceinline__ int2 work_range(const Work& w) { return w.seg ? *w.seg : make_int2(w.first, w.count); }
template <typename R> __device__ __forceinline__ const LatDesc<R>* work_member(const Work& w, const LatDesc<R>* descs, int member) {
    return w.seg ? descs + member : descs;
}

// ------------------------------------------------------------------ stage
// One RK3 stage (low-storage form of the reference's integrator):
//   S=1:  A = Z0;                    U1 = exp(eps/4 Z0) U0
//   S=2:  A = 8/9 Z1 - 17/36 A;      U2 = exp(eps A) U1
//   S=3:                             U3 = exp(eps (3/4 Z2 - A)) U2
// which equals GradientFlow.cpp:27-50 term by term.  Input and output are
// different buffers of the ring (every thread reads neighbours of the input).
template <typename R, int S> __device__ __forceinline__ const cplx<R>* stage_in(const LatDesc<R>* d) { return S == 1 ? d->U0 : (S == 2 ? d->U1 : d->U2); }
template <typename R, int S> __device__ __forceinline__ cplx<R>* stage_out(const LatDesc<R>* d) { return S == 1 ? d->U1 : (S == 2 ? d->U2 : d->U0); }
template <typename R, int S> __device__ __forceinline__ R* stage_free(const LatDesc<R>* d) { return reinterpret_cast<R*>(S == 1 ? d->U2 : (S == 2 ? d->U0 : d->U1)); }

// accumulator, exponential and link update of link (s, mu) with force Z and
// link u.  The integrator's coefficients and eps are applied in double for
// both precisions: in float they round by up to 2e-8 of themselves, the same
// way at every step, which is a flow time off by as much.
template <typename R, int S>
__device__ __forceinline__ void update_link(R* A, cplx<R>* Uout, double eps, int V, int s, int mu, const alg<R>& Z, const su3<R>& u) {
    alg<double> X = alg_cast<double>(Z);
    if (S == 1) {
        store_alg(A, V, mu, s, Z);
        X = alg_scale(0.25 * eps, X);
    } else if (S == 2) {
        X = alg_axpby(8.0 / 9.0, X, -17.0 / 36.0, alg_cast<double>(load_alg(A, V, mu, s)));
        store_alg(A, V, mu, s, alg_cast<R>(X));
        X = alg_scale(eps, X);
    } else {
        X = alg_axpby(3.0 / 4.0, X, -1.0, alg_cast<double>(load_alg(A, V, mu, s)));
        X = alg_scale(eps, X);
    }
    // the stored link is the full product (rebuilding its third row from
    // the first two would let their rounding drift into it step after step)
    store_link(Uout, V, mu, s, exp_times(X, u));
}

// Staple form: large FP64 lattices, and middle-sized ones of either precision
// (stage_form); PARTS as in staple_sum.
// Persistent: blocks stride over one segment of the tile list (seg = first
// tile, count); tile = (lattice, first site).
// A tile of T threads (T a multiple of 128) covers T/4 consecutive sites with
// all four directions: warp w handles mu = w % 4 for the 32 sites of group
// w / 4, so the four link directions of a site range are read together and
// every load of a warp covers 32 consecutive sites.
template <typename R> struct StageMaxThreads { static constexpr int value = LGF_STAGE_MAXT_F; };
template <> struct StageMaxThreads<double> { static constexpr int value = LGF_STAGE_MAXT_D; };

template <typename R, int S, bool PARTS>
__global__ void __launch_bounds__(StageMaxThreads<R>::value, LGF_STAGE_MINB) k_rk3_stage(const LatDesc<R>* __restrict__ descs, const int2* __restrict__ tiles,
                                                   Work work) {
    const int2 r = work_range(work);  // this launch's tiles: tiles[r.x, r.x + r.y)
    for (int ti = r.x + blockIdx.x; ti < r.x + r.y; ti += gridDim.x) {
        const int2 tile = tiles[ti];
        const LatDesc<R>* d = work_member(work, descs, tile.x);
        const Geom g = d->g;
        const int mu = (threadIdx.x >> 5) & 3;
        const int s = tile.y + ((threadIdx.x >> 7) << 5) + (threadIdx.x & 31);
        if (s >= g.V) continue;
        const cplx<R>* Uin = stage_in<R, S>(d);
        cplx<R>* Uout = stage_out<R, S>(d);
        R* A = d->A;
        const double eps = d->eps;
        const Coord c = site_coord(g, s);
        su3<R> u;
        const alg<R> Z = flow_gradient<R, PARTS>(Uin, g, s, c, mu, u);
        update_link<R, S>(A, Uout, eps, g.V, s, mu, Z, u);
    }
}

// Split form: lattices of up to one 32-site tile per SM.  With one warp per
// direction and tile an SM's schedulers hold a warp each, and a stage is the
// latency of one thread's six staples; here three warps take two staples each
// and the first adds their sums (in a fixed order) and updates the link.
// 8^4 FP64 22.6 -> 20 us per step (19 with the range by value, Work), FP32
// 18.5 -> 17.5 (16.5).  Above the line an SM with two tiles would run them in
// turn, and the staple form runs them side by side.
// Where a group's small lattices have more tiles than that, the staple form
// with the same grouping of the sum (PARTS) takes them, so that the bits are
// those the lattice gives alone: 64 x 8^4 batched, 200 steps, FP32 84 -> 78 ms
// on the device, FP64 117 -> 113 with the launch's best block size (the split
// kernel itself, a tile per SM at a time, took 1.5 times as long).
constexpr int SPLIT_SITES = 32, SPLIT_THREADS = 12 * SPLIT_SITES;
constexpr long long SPLIT_MAX_SITES = 148 * SPLIT_SITES;
template <typename R, int S>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) k_rk3_split(const LatDesc<R>* __restrict__ descs, const int2* __restrict__ tiles,
                                                               Work work) {
    __shared__ typename vec2_of<R>::type part_sum[2][9][4 * SPLIT_SITES];
    const int2 r = work_range(work);
    const int lane = threadIdx.x & 31, mu = (threadIdx.x >> 5) & 3, part = threadIdx.x >> 7, column = threadIdx.x & 127;
    for (int ti = r.x + blockIdx.x; ti < r.x + r.y; ti += gridDim.x) {
        const int2 tile = tiles[ti];
        const LatDesc<R>* d = work_member(work, descs, tile.x);
        const Geom g = d->g;
        const int s = tile.y + lane;
        const bool in = s < g.V;
        const cplx<R>* Uin = stage_in<R, S>(d);
        su3<R> sum;
        su3_zero(sum);
        if (in) {
            const Coord c = site_coord(g, s);
            const Dir dm = dir_of(g, c, mu);
            const int nu = part + (part >= mu ? 1 : 0);
            add_staples(sum, Uin, g, s, mu, dm, fwd(s, dm), nu, sel4(nu, c.x[0], c.x[1], c.x[2], c.x[3]));
            if (part > 0) {
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    typename vec2_of<R>::type v;
                    v.x = sum.m[k].re;
                    v.y = sum.m[k].im;
                    part_sum[part - 1][k][column] = v;
                }
            }
        }
        __syncthreads();
        if (in && part == 0) {
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const typename vec2_of<R>::type v = part_sum[0][k][column], w = part_sum[1][k][column];
                sum.m[k] = cmk<R>((sum.m[k].re + v.x) + w.x, (sum.m[k].im + v.y) + w.y);
            }
            const su3<R> u = load_link(Uin, g.V, mu, s);
            update_link<R, S>(d->A, stage_out<R, S>(d), d->eps, g.V, s, mu, ta_of_product(u, sum, R(-0.5)), u);
        }
        __syncthreads();
    }
}

// Plaquette form: FP32 lattices above the small ones, FP64 ones that L2 holds.
//
// The force of link (x, mu) sums the six plaquettes that contain the link,
// projected: Z = -i sum_nu F[W_+nu] + F[W_-nu] with W based at x and starting
// along mu.  Every plaquette belongs to four links.  With its projection
// P_mn(y) = F[m(y) n(y+m) (n(y) m(y+n))^dag] at its lowest corner (m < n), and
// T_d the covariant shift of a projection (shift()),
//     link (x, m):  F[W_+n] + F[W_-n] =   P_mn(x) - T_n P_mn(x)
//     link (x, n):  F[W_+m] + F[W_-m] = -(P_mn(x) - T_m P_mn(x)),
// so a site's six plaquettes (two products and a projection each) and twelve
// shifts replace its 24 staples: 4600 instead of 6500 operations per site and
// stage.  The plaquettes make a launch of their own and go to the ring's free
// buffer (stage S reads U_{S-1}, writes U_S; six fields of 8 reals take two
// thirds of the third), which costs 384 (FP64: 768) bytes of traffic per site.
// FP32, bound by instruction issue, gains: one B200, us per step (3 stages),
// 24^3x48 803 -> 661, 32^4 1251 -> 1012, 48^4 6900 -> 5600, 16^4 89 -> 76,
// 6x10x14x18 35 -> 31.
// FP64 gains where L2 holds what is read again, links and projections, 960
// bytes per site: 16^4 138 -> 119, 32x16^3 272 -> 237, 12^4 53 -> 49.  Beyond
// it is bound by that traffic (24^3x48: plaquettes 153 us at 0.49 of the FP64
// pipe, update 278 us at 0.45 with DRAM at 5 TB/s): 24^3x48 1197 -> 1205, 48^4
// 10160 -> 11250; keeping a chunk of x0 slices' plaquettes in L2 with a launch
// per chunk was slower still (1350 in chunks of 256 MB, 1570 of 64 MB).
constexpr int PLAQ_SITES = 32;    // sites of a plaquette tile: a warp per plane
constexpr int UPDATE_SITES = 32;  // sites of an update tile: a warp per direction
template <typename R> __device__ __forceinline__ R* plaq_field(R* K, int p, int s) {
    return K + ((size_t)(s / LAYOUT_BLOCK) * 6 + p) * FIELD_REALS + (s % LAYOUT_BLOCK) * (16 / sizeof(R));
}
// index of plane (a, b), a < b, in the order 01 02 03 12 13 23
__host__ __device__ __forceinline__ int plane_index(int a, int b) { return a == 0 ? b - 1 : a + b; }

template <typename R>
__device__ __forceinline__ void plaquette_at(const cplx<R>* __restrict__ U, R* __restrict__ K, const Geom& g, int s, const Coord& c, int p) {
    const int m = c_plane_mu[p], n = c_plane_nu[p];
    const int xpm = fwd(s, dir_of(g, c, m)), xpn = fwd(s, dir_of(g, c, n));
    const su3<R> a = mul_nn_su3(load_link(U, g.V, m, s), load_link(U, g.V, n, xpm));
    const su3<R> b = mul_nn_su3(load_link(U, g.V, n, s), load_link(U, g.V, m, xpn));
    put_field(plaq_field(K, p, s), leaf<R>(a, b, R(1)));
}

// Z(x, mu) from the plaquettes, in the coordinates of an su(3) element:
// X = -i F has (Im X00, Im X11) = -(F00, F11) and X_ij = (Im F_ij, -Re F_ij)
template <typename R>
__device__ __forceinline__ alg<R> force_at(const cplx<R>* __restrict__ U, const R* __restrict__ K, const Geom& g, int s, const Coord& c,
                                           int mu) {
    alg<R> f;
#pragma unroll
    for (int k = 0; k < 8; ++k) f.v[k] = R(0);
    const int n1 = (mu + 1) & 3, n2 = (mu + 2) & 3, n3 = (mu + 3) & 3;
    auto plane = [&](int nu) { return mu < nu ? plane_index(mu, nu) : plane_index(nu, mu); };
    auto H = [&](int nu, int at) { return get_field<R, true>(plaq_field(K, plane(nu), at)); };
    const int b1 = bwd(s, dir_of(g, c, n1)), b2 = bwd(s, dir_of(g, c, n2)), b3 = bwd(s, dir_of(g, c, n3));
    auto add = [&](int nu, const alg<R>& k0, const alg<R>& t) {
        const R sg = mu < nu ? R(1) : R(-1);
#pragma unroll
        for (int k = 0; k < 8; ++k) f.v[k] = fma(sg, k0.v[k] - t.v[k], f.v[k]);
    };
    // the next direction's loads are issued before this one's shift
    const su3<R> l1 = load_link(U, g.V, n1, b1);
    const alg<R> h1 = H(n1, b1);
    const su3<R> l2 = load_link(U, g.V, n2, b2);
    const alg<R> h2 = H(n2, b2);
    const alg<R> k1 = H(n1, s);
    add(n1, k1, shift(h1, l1));
    const su3<R> l3 = load_link(U, g.V, n3, b3);
    const alg<R> h3 = H(n3, b3);
    const alg<R> k2 = H(n2, s);
    add(n2, k2, shift(h2, l2));
    const alg<R> k3 = H(n3, s);
    add(n3, k3, shift(h3, l3));
    alg<R> z;
    z.v[0] = -f.v[0];
    z.v[1] = -f.v[1];
#pragma unroll
    for (int k = 2; k < 8; k += 2) {
        z.v[k] = f.v[k + 1];
        z.v[k + 1] = -f.v[k];
    }
    return z;
}

// FP32: 24 warps of 80 registers per SM (30 of 64 registers: 16^4 5% slower).
// FP64: 12 of 158, which leave the compiler room to issue a plaquette's loads
// together (18 of 96: 16^4 124 us per step instead of 119).
template <typename R> __host__ __device__ constexpr int plaq_blocks() { return sizeof(R) == sizeof(float) ? 4 : 2; }
template <typename R, int S>
__global__ void __launch_bounds__(6 * PLAQ_SITES, plaq_blocks<R>()) k_rk3_plaquettes(const LatDesc<R>* __restrict__ descs, const int2* __restrict__ tiles,
                                                                     Work work) {
    const int2 r = work_range(work);  // this launch's tiles: tiles[r.x, r.x + r.y)
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int ti = r.x + blockIdx.x; ti < r.x + r.y; ti += gridDim.x) {
        const int2 tile = tiles[ti];
        const LatDesc<R>* d = work_member(work, descs, tile.x);
        const Geom g = d->g;
        const int s = tile.y + (w / 6) * 32 + lane;
        if (s < g.V) plaquette_at<R>(stage_in<R, S>(d), stage_free<R, S>(d), g, s, site_coord(g, s), w % 6);
    }
}

// FP32: 20 warps of 96 registers per SM (24 of 80 with each load beside its
// shift: 32^4 1030 us per step instead of 1012; 16 of 127: 1037).  FP64: 16 of
// 128 (20 of 96 spill: 16^4 134 instead of 119; 12 of 168: 124).
template <typename R> __host__ __device__ constexpr int update_blocks() { return sizeof(R) == sizeof(float) ? 5 : 4; }
template <typename R, int S>
__global__ void __launch_bounds__(4 * UPDATE_SITES, update_blocks<R>()) k_rk3_update(const LatDesc<R>* __restrict__ descs, const int2* __restrict__ tiles,
                                                                   Work work) {
    const int2 r = work_range(work);
    const int mu = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int ti = r.x + blockIdx.x; ti < r.x + r.y; ti += gridDim.x) {
        const int2 tile = tiles[ti];
        const LatDesc<R>* d = work_member(work, descs, tile.x);
        const Geom g = d->g;
        const int s = tile.y + lane;
        if (s >= g.V) continue;
        const cplx<R>* Uin = stage_in<R, S>(d);
        const alg<R> Z = force_at<R>(Uin, stage_free<R, S>(d), g, s, site_coord(g, s), mu);
        update_link<R, S>(d->A, stage_out<R, S>(d), d->eps, g.V, s, mu, Z, load_link(Uin, g.V, mu, s));
    }
}

// Whether a lattice's stages take the plaquette form.  Small lattices do not:
// the two short launches cost more than the operations they save.  FP32, us per
// step in the staple form with a sum per direction (PARTS), with one sum for
// all, and in the plaquette form:
//    4800  18.4  20.5  22.6      8192  18.6  21    24        9600  22.5  24.6  26.6
//   12000  22.6  24.7  26.6     13824  23.2  24.6  27       14400  31.8  34.8  29.3
//   15120        34.8  30.7     20736        37    34.8
// so the line is one wave of the staple form: three 32-site tiles per SM.  In
// batches of eight and more such lattices the plaquette form would be 0 to 3%
// faster (16 x 13440 sites, 100 steps, 34.5 against 35.7 ms; 39.8 with one sum),
// in smaller ones slower (2 of them 6.3 against 5.5).
// FP64: 16384 sites 41 (staple, PARTS 41) against 43, 20736: 53 against 49.  Nor
// do FP64 lattices past L2 (196608 sites: 365 against 379; 276480, 331776,
// 442368: equal within the runs' spread; 48^4 11% slower).  The rule reads the
// lattice alone, so a lattice gives the same bits in every group.
constexpr int STAPLE_MAX_SITES_FP32 = 3 * 148 * 32;
constexpr int PLAQ_MIN_SITES_FP64 = 18432, PLAQ_MAX_SITES_FP64 = 200000;
template <typename R> __host__ __device__ __forceinline__ bool plaquette_stage(const Geom& g) {
    return sizeof(R) == sizeof(float) ? g.V > STAPLE_MAX_SITES_FP32 : g.V >= PLAQ_MIN_SITES_FP64 && g.V <= PLAQ_MAX_SITES_FP64;
}
// The forms: staple with one sum for all directions (FP64: above the split
// form 26.6 us per step against 28.7 to 30.7 with PARTS), plaquette, split, and
// staple with a sum per direction (FP32, and split lattices in large groups).
constexpr int FORM_STAPLE = 0, FORM_PLAQUETTE = 1, FORM_SPLIT = 2, FORM_PARTS = 3, FORMS = 4;
template <typename R> __host__ __device__ __forceinline__ int stage_form(const Geom& g) {
    if (g.V <= SPLIT_MAX_SITES) return FORM_SPLIT;
    if (plaquette_stage<R>(g)) return FORM_PLAQUETTE;
    return sizeof(R) == sizeof(float) ? FORM_PARTS : FORM_STAPLE;
}

template <typename R> __device__ __forceinline__ void store_alg_as_antiherm(double2* dst, const alg<R>& z) {
    const double v0 = z.v[0], v1 = z.v[1];
    dst[0] = make_double2(0.0, v0);
    dst[4] = make_double2(0.0, v1);
    dst[8] = make_double2(0.0, -(v0 + v1));
    dst[1] = make_double2(z.v[2], z.v[3]);
    dst[3] = make_double2(-(double)z.v[2], z.v[3]);
    dst[2] = make_double2(z.v[4], z.v[5]);
    dst[6] = make_double2(-(double)z.v[4], z.v[5]);
    dst[5] = make_double2(z.v[6], z.v[7]);
    dst[7] = make_double2(-(double)z.v[6], z.v[7]);
}
template <typename R> __device__ __forceinline__ void store_alg_as_herm(double2* dst, const alg<R>& f) {
    const double v0 = f.v[0], v1 = f.v[1];
    dst[0] = make_double2(v0, 0.0);
    dst[4] = make_double2(v1, 0.0);
    dst[8] = make_double2(-(v0 + v1), 0.0);
    dst[1] = make_double2(f.v[2], f.v[3]);
    dst[3] = make_double2(f.v[2], -(double)f.v[3]);
    dst[2] = make_double2(f.v[4], f.v[5]);
    dst[6] = make_double2(f.v[4], -(double)f.v[5]);
    dst[5] = make_double2(f.v[6], f.v[7]);
    dst[7] = make_double2(f.v[6], -(double)f.v[7]);
}

constexpr int MEAS_SITES = 32;  // sites per measurement block (x) ; planes in y

// Offset within its x0 slice of lane l's site in measurement chunk c: a tile is
// 32 consecutive sites of the slice.  The geometry is a fixed function of the
// lattice shape, so the grouping of the partial sums (and every result bit)
// does not depend on tile shapes or batch partners.
__host__ __device__ __forceinline__ int meas_site_offset(int c, int l) { return c * MEAS_SITES + l; }
#ifndef LGF_MEAS_SMEM_ACC
#define LGF_MEAS_SMEM_ACC 1
#endif
constexpr int MEAS_ACC_STRIDE = MEAS_SITES * 12;  // one column per thread of a 12-warp block
template <typename R> __device__ __forceinline__ R SmemAcc<R>::get(int k) const { return p[k * MEAS_ACC_STRIDE]; }
template <typename R> __device__ __forceinline__ void SmemAcc<R>::set(int k, R x) { p[k * MEAS_ACC_STRIDE] = x; }
template <typename R> constexpr bool meas_smem_acc() { return LGF_MEAS_SMEM_ACC && sizeof(R) == sizeof(double); }

// A path matrix parked in the thread's own shared-memory column until it is
// extended by one more link.  Only its first two rows are kept when the
// extension rebuilds the third (mul_nn_su3 / mul_na_su3 read rows 0 and 1 of
// their left operand), so a parked path is exactly the one put there.
constexpr int MEAS_STASH_ENTRIES = 6;
template <typename R, int ENTRIES = MEAS_STASH_ENTRIES> struct PathStash {
    typename vec2_of<R>::type* p;  // entry k at p[k * MEAS_ACC_STRIDE]
    __device__ __forceinline__ void put(const su3<R>& P) const {
#pragma unroll
        for (int k = 0; k < ENTRIES; ++k) {
            p[k * MEAS_ACC_STRIDE].x = P.m[k].re;
            p[k * MEAS_ACC_STRIDE].y = P.m[k].im;
        }
    }
    __device__ __forceinline__ su3<R> get() const {
        su3<R> P;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            if (k < ENTRIES) {
                const typename vec2_of<R>::type v = p[k * MEAS_ACC_STRIDE];
                P.m[k] = cmk<R>(v.x, v.y);
            } else {
                P.m[k] = cmk<R>(R(0), R(0));  // never read: the next product rebuilds the row
            }
        }
        return P;
    }
};

// Shared memory of one measurement block: the straight lines of length 2 and
// 3 from each of its 32 sites in the 8 signed directions (every plane and
// quadrant of the site reuses them), then the per-plane results.  With FILE
// the paths keep all nine entries, and there is room for one parked path.
template <typename R, bool FILE = false> struct MeasSmem {
    static constexpr int ENTRIES = FILE ? 9 : MEAS_STASH_ENTRIES, PARKED = FILE ? 1 : 2;
    union {
        R line[8][2][2 * ENTRIES][MEAS_SITES];  // [2*dir + (sign<0)][length-2][real of entry][site]
        struct {                       // after the lines are dead: the second quadrant half's sums
            alg<R> G[6][MEAS_SITES];
            alg<R> Fh[6][MEAS_SITES];
        } part;
    };
    R acc[meas_smem_acc<R>() ? 16 : 1][meas_smem_acc<R>() ? MEAS_ACC_STRIDE : 1];  // G, Fhat columns (LGF_MEAS_SMEM_ACC)
    typename vec2_of<R>::type stash[PARKED][ENTRIES][MEAS_ACC_STRIDE];  // parked paths per thread (PathStash)
    alg<R> F[6][MEAS_SITES];          // improved F per plane
    double E[6][MEAS_SITES];
};

// What a measurement pass may write besides the sums (single-lattice calls;
// all null in the flow): e, q the site densities; swap: e with the improved F
// and q with the clover F (ImprovedEnergyDensity.cpp:13-20,
// UnImprovedTopologicalCharge.cpp:11-16); dbg_*: F and F^ as Hermitian 3x3
// matrices per (site, plane).
struct MeasSites {
    double* e;
    double* q;
    int swap;
    double2* dbg_clover;
    double2* dbg_improved;
};

// A line is only ever extended (the left operand of a product that rebuilds
// the third row), so like a parked path it keeps its first two rows.
template <typename R, bool FILE>
__device__ __forceinline__ void store_line(MeasSmem<R, FILE>* sm, int sdir, int len, int lane, const su3<R>& L) {
#pragma unroll
    for (int k = 0; k < MeasSmem<R, FILE>::ENTRIES; ++k) {
        sm->line[sdir][len - 2][2 * k][lane] = L.m[k].re;
        sm->line[sdir][len - 2][2 * k + 1][lane] = L.m[k].im;
    }
}
template <typename R, bool FILE>
__device__ __forceinline__ su3<R> load_line(const MeasSmem<R, FILE>* sm, int sdir, int len, int lane) {
    su3<R> L;
#pragma unroll
    for (int k = 0; k < 9; ++k)
        L.m[k] = k < MeasSmem<R, FILE>::ENTRIES
                     ? cmk<R>(sm->line[sdir][len - 2][2 * k][lane], sm->line[sdir][len - 2][2 * k + 1][lane])
                     : cmk<R>(R(0), R(0));  // never read: the next product rebuilds the row
    return L;
}

// Quadrants [qa, qb) of plane (mu, nu) at the thread's site, using the
// block's shared lines: G = the sum of the 1x1 leaves' projections, Fhat =
// the weighted sum of the other shapes' (see the comment above Plane for the
// leaf decomposition).  The clover F is G/4 and the improved F is
// Fhat + 19/36 G.  With a b-fold path written as its steps (n = sn nu,
// m = sm mu), the twelve paths of a quadrant are
//   Pn(a,1) = n m^a        (a chain: each extends the one before by m)
//   Pm(1,b) = m n^b        (a chain along n)
//   Pm(a,1) = line_m(a) n,  Pn(1,b) = line_n(b) m   (from the shared lines)
//   Pn(2,2) = Pn(1,2) m,    Pm(2,2) = Pm(2,1) n
// 12 matrix products and 14 global link loads per quadrant; the paths that
// are extended after other work are parked in the thread's shared-memory
// column (PathStash: Pm(1,1), Pm(2,1), Pn(1,2)), and the leaves are added in
// the order (1,1) | (2,1), (3,1), (1,2), (1,3), (2,2).  With FILE, Pm(2,1) is
// formed again instead (one product and one load more).
template <typename R, bool FILE, typename Acc>
__device__ __forceinline__ void plane_fields_body(const cplx<R>* __restrict__ U, const Geom& g, int s, const Coord& c,
                                                  int mu, int nu, const MeasSmem<R, FILE>* sm, int lane, int qa, int qb,
                                                  Acc G, Acc Fhat, PathStash<R, MeasSmem<R, FILE>::ENTRIES> sa,
                                                  PathStash<R, MeasSmem<R, FILE>::ENTRIES> sb) {
    Plane<R, R, FILE> P;
    P.U = U;
    P.V = g.V;
    P.mu = mu;
    P.nu = nu;
    P.dm = dir_of(g, c, mu);
    P.dn = dir_of(g, c, nu);
    const PlanePos x0 = {s, P.dm.x, P.dn.x};
    const R k12 = R(-4.0 / 45.0), k13 = R(1.0 / 120.0), k22 = R(1.0 / 144.0);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        G.set(k, R(0));
        Fhat.set(k, R(0));
    }
#pragma unroll 1
    for (int q = qa; q < qb; ++q) {
        const int sm_ = (q == 0 || q == 1) ? 1 : -1;
        const int sn = (q == 0 || q == 2) ? 1 : -1;
        const R sg = (q == 0 || q == 3) ? R(1) : R(-1);
        const int sdm = 2 * mu + (sm_ < 0 ? 1 : 0), sdn = 2 * nu + (sn < 0 ? 1 : 0);
        // (1,1)
        PlanePos pn = x0;
        su3<R> Pn = P.step(pn, false, sn);
        P.ext(Pn, pn, true, sm_);  // Pn(1,1)
        PlanePos pm = x0;
        su3<R> Pm = P.step(pm, true, sm_);
        P.ext(Pm, pm, false, sn);  // Pm(1,1), pm at x + m + n
        leaf_acc(Pn, Pm, sg, G);
        sa.put(Pm);
        // (2,1)
        P.ext(Pn, pn, true, sm_);  // Pn(2,1)
        PlanePos p21 = x0;
        P.advance(p21, true, sm_, 2);
        Pm = load_line(sm, sdm, 2, lane);
        P.ext(Pm, p21, false, sn);  // Pm(2,1), p21 at x + 2m + n
        leaf_acc(Pn, Pm, sg * k12, Fhat);
        if (!FILE) sb.put(Pm);
        // (3,1)
        P.ext(Pn, pn, true, sm_);  // Pn(3,1)
        PlanePos p31 = x0;
        P.advance(p31, true, sm_, 3);
        Pm = load_line(sm, sdm, 3, lane);
        P.ext(Pm, p31, false, sn);  // Pm(3,1)
        leaf_acc(Pn, Pm, sg * k13, Fhat);
        // (1,2)
        Pm = sa.get();
        P.ext(Pm, pm, false, sn);  // Pm(1,2)
        PlanePos p12 = x0;
        P.advance(p12, false, sn, 2);
        Pn = load_line(sm, sdn, 2, lane);
        P.ext(Pn, p12, true, sm_);  // Pn(1,2), p12 at x + 2n + m
        leaf_acc(Pn, Pm, sg * k12, Fhat);
        sa.put(Pn);
        // (1,3)
        P.ext(Pm, pm, false, sn);  // Pm(1,3)
        PlanePos p13 = x0;
        P.advance(p13, false, sn, 3);
        Pn = load_line(sm, sdn, 3, lane);
        P.ext(Pn, p13, true, sm_);  // Pn(1,3)
        leaf_acc(Pn, Pm, sg * k13, Fhat);
        // (2,2)
        Pn = sa.get();
        P.ext(Pn, p12, true, sm_);  // Pn(2,2)
        if (FILE) {
            p21 = x0;
            P.advance(p21, true, sm_, 2);
            Pm = load_line(sm, sdm, 2, lane);
            P.ext(Pm, p21, false, sn);  // Pm(2,1)
        } else {
            Pm = sb.get();
        }
        P.ext(Pm, p21, false, sn);  // Pm(2,2)
        leaf_acc(Pn, Pm, sg * k22, Fhat);
    }
}

template <typename R, bool FILE>
__device__ __forceinline__ void plane_fields_smem(const cplx<R>* __restrict__ U, const Geom& g, int s, const Coord& c,
                                                  int mu, int nu, MeasSmem<R, FILE>* sm, int lane, int qa, int qb,
                                                  alg<R>& Greg, alg<R>& Fhreg) {
    const int column = threadIdx.y * MEAS_SITES + lane;
    const PathStash<R, MeasSmem<R, FILE>::ENTRIES> sa{&sm->stash[0][0][column]},
        sb{&sm->stash[MeasSmem<R, FILE>::PARKED - 1][0][column]};  // (unused with FILE)
    if constexpr (meas_smem_acc<R>()) {
        R* col = &sm->acc[0][column];
        const SmemAcc<R> G{col}, Fhat{col + 8 * MEAS_ACC_STRIDE};
        plane_fields_body<R, FILE>(U, g, s, c, mu, nu, sm, lane, qa, qb, G, Fhat, sa, sb);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            Greg.v[k] = G.get(k);
            Fhreg.v[k] = Fhat.get(k);
        }
    } else {
        plane_fields_body<R, FILE>(U, g, s, c, mu, nu, sm, lane, qa, qb, RegAcc<R>{Greg}, RegAcc<R>{Fhreg}, sa, sb);
    }
}

// Measurement of small lattices in one launch (small_measure, lgf_measure.cuh).
// Tile = (lattice, x0 slice, chunk of 32 consecutive sites of the slice); 12
// warps: warp y takes plane y % 6 and two of the four quadrants (part y / 6).
// Phase 0: the block's lines (a warp per signed direction) into shared memory.
// Phase 1: the quadrant sums of every (site, plane); the second part's sums
// meet the first's in the (then dead) line storage, in a fixed order, for F
// and F^.  Phase 2: the six planes meet in shared memory for e(x) and q(x);
// the tile's sums go to the lattice's partial[slice * nchunk + chunk].
//   e(x) = sum_{mu<nu} ReTr(F F)                 (EnergyDensity.cpp:13-20)
//   q(x) = ReTr(F^32 F^01) + ReTr(F^31 F^20) + ReTr(F^30 F^12)
//        = -T(23,01) + T(13,02) - T(03,12),  T(a,b) = ReTr(F^a F^b)
//                                             (TopologicalCharge.cpp:11-16)
constexpr int MEAS_WARPS = 12;
template <typename R, bool OUT, bool FILE>
__device__ __forceinline__ void measure_tile(MeasSmem<R, FILE>* sm, const cplx<R>* __restrict__ U, const Geom& g, int slice, int chunk,
                                             double2* __restrict__ partial, int nchunk, const MeasSites& out) {
    const int lane = threadIdx.x, w = threadIdx.y, p = w % 6, part = w / 6;
    const int off = meas_site_offset(chunk, lane);
    const bool valid = off < g.Vs;
    const int s = slice * g.Vs + (valid ? off : 0);
    const Coord c = site_coord(g, s);
    // phase 0: lines of length 2 and 3 in the 8 signed directions
    if (w < 8) {
        const int dir = w >> 1, sign = (w & 1) ? -1 : 1;
        Plane<R, R, FILE> L;
        L.U = U;
        L.V = g.V;
        L.mu = dir;
        L.nu = dir;
        L.dm = dir_of(g, c, dir);
        L.dn = L.dm;
        PlanePos y = {s, L.dm.x, L.dm.x};
        su3<R> acc = L.step(y, true, sign);
        L.ext(acc, y, true, sign);
        store_line(sm, w, 2, lane, acc);
        L.ext(acc, y, true, sign);
        store_line(sm, w, 3, lane, acc);
    }
    __syncthreads();
    // phase 1: this thread's plane and quadrants
    alg<R> G, Fh;
    if (FILE || valid) plane_fields_smem<R, FILE>(  // (file-order loads need the whole warp)
        U, g, s, c, c_plane_mu[p], c_plane_nu[p], sm, lane, 2 * part, 2 * part + 2, G, Fh);
    __syncthreads();  // every warp is done with the lines
    if (part == 1 && valid) {
        sm->part.G[p][lane] = G;
        sm->part.Fh[p][lane] = Fh;
    }
    __syncthreads();
    if (part == 0 && valid) {
        const alg<R> G1 = sm->part.G[p][lane], F1 = sm->part.Fh[p][lane];
        alg<R> F11;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            G.v[k] += G1.v[k];
            Fh.v[k] += F1.v[k];
            F11.v[k] = R(0.25) * G.v[k];
            Fh.v[k] = fma(R(19.0 / 36.0), G.v[k], Fh.v[k]);
        }
        if (OUT) {
            if (out.dbg_clover) store_alg_as_herm(out.dbg_clover + ((size_t)s * 6 + p) * 9, F11);
            if (out.dbg_improved) store_alg_as_herm(out.dbg_improved + ((size_t)s * 6 + p) * 9, Fh);
            if (out.swap) {
                const alg<R> z = F11;
                F11 = Fh;
                Fh = z;
            }
        }
        sm->F[p][lane] = Fh;
        sm->E[p][lane] = retr_hh(F11, F11);
    }
    __syncthreads();
    // phase 2: the site's e(x), q(x) and the tile's sums
    if (w == 0) {
        double e = 0.0, q = 0.0;
        if (valid) {
            e = ((sm->E[0][lane] + sm->E[1][lane]) + (sm->E[2][lane] + sm->E[3][lane])) +
                (sm->E[4][lane] + sm->E[5][lane]);
            q = -retr_hh(sm->F[5][lane], sm->F[0][lane]) + retr_hh(sm->F[4][lane], sm->F[1][lane]) -
                retr_hh(sm->F[2][lane], sm->F[3][lane]);
            if (OUT) {
                if (out.e) out.e[s] = e;
                if (out.q) out.q[s] = q;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            e += __shfl_xor_sync(0xffffffffu, e, o);
            q += __shfl_xor_sync(0xffffffffu, q, o);
        }
        if (lane == 0) partial[slice * nchunk + chunk] = make_double2(e, q);
    }
}

template <typename R, bool OUT>
__global__ void __launch_bounds__(MEAS_SITES * MEAS_WARPS, 1) k_measure(const LatDesc<R>* __restrict__ descs,
                                                                       const int4* __restrict__ mtiles,
                                                                       Work work, MeasSites out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MeasSmem<R>* sm = reinterpret_cast<MeasSmem<R>*>(smem_raw);
    const int2 r = work_range(work);  // this launch's tiles: mtiles[r.x, r.x + r.y)
    for (int ti = r.x + blockIdx.x; ti < r.x + r.y; ti += gridDim.x) {
        const int4 tile = mtiles[ti];
        const LatDesc<R>* d = work_member(work, descs, tile.x);
        const Geom g = d->g;
        measure_tile<R, OUT, false>(sm, d->U0, g, tile.y, tile.z, d->partial, d->nchunk, out);
        __syncthreads();
    }
}

// Dynamic shared memory of k_measure<R> (above 48 KB: raised with the kernel's
// attribute before the first launch).
template <typename R, bool FILE = false> inline size_t measure_smem_bytes() { return sizeof(MeasSmem<R, FILE>); }

constexpr int RED_THREADS = 256;

// Slice sums and totals in fixed order (deterministic run to run).  One block
// per (lattice, slice) entry of rtiles: thread i sums chunks i, i+256, ...
// sequentially, then a fixed binary tree.  The block that finishes a lattice's
// last slice (a counter beside its slot that wraps back to 0) sums the slices
// the same way; which block that is changes no order.  Result slot layout per
// measurement: [E, Q, E_slice[N0], Q_slice[N0]] at meas + (*slot) * (2 + 2 N0).
// One launch instead of two saves 2 us of an 8^4 measurement's 35.
__device__ __forceinline__ double2 block_sum(double e, double q, double* se, double* sq) {
    se[threadIdx.x] = e;
    sq[threadIdx.x] = q;
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            se[threadIdx.x] += se[threadIdx.x + w];
            sq[threadIdx.x] += sq[threadIdx.x + w];
        }
        __syncthreads();
    }
    return make_double2(se[0], sq[0]);
}

template <typename R>
__global__ void __launch_bounds__(RED_THREADS) k_reduce(const LatDesc<R>* __restrict__ descs, const int2* __restrict__ rtiles,
                                                        const int* __restrict__ nrtiles, Work work) {
    __shared__ double se[RED_THREADS], sq[RED_THREADS];
    __shared__ bool last;
    const double inv4pi2 = 1.0 / (4.0 * 3.14159265358979323846 * 3.14159265358979323846);
    const int n = work.seg ? *nrtiles : work.count;
    for (int ti = blockIdx.x; ti < n; ti += gridDim.x) {
        const int2 tile = rtiles[ti];
        const LatDesc<R>* d = work_member(work, descs, tile.x);
        const int t = tile.y, N0 = d->g.n[0], nchunk = d->nchunk;
        double e = 0.0, q = 0.0;
        for (int j = threadIdx.x; j < nchunk; j += RED_THREADS) {
            const double2 v = d->partial[t * nchunk + j];
            e += v.x;
            q += v.y;
        }
        const double2 sum = block_sum(e, q, se, sq);
        if (threadIdx.x == 0) {
            double* o = d->meas + (size_t)(*d->slot) * (2 + 2 * N0);
            o[2 + t] = sum.x / (double)d->g.Vs;
            o[2 + N0 + t] = sum.y * inv4pi2;
            d->slice_sums[t] = sum;
            __threadfence();
            last = atomicInc(reinterpret_cast<unsigned int*>(d->slot + 1), (unsigned int)(N0 - 1)) == (unsigned int)(N0 - 1);
        }
        __syncthreads();
        if (last) {
            __threadfence();
            e = q = 0.0;
            for (int j = threadIdx.x; j < N0; j += RED_THREADS) {
                const double2 v = __ldcg(d->slice_sums + j);
                e += v.x;
                q += v.y;
            }
            const double2 all = block_sum(e, q, se, sq);
            if (threadIdx.x == 0) {
                double* o = d->meas + (size_t)(*d->slot) * (2 + 2 * N0);
                o[0] = all.x * (1.0 / (double)d->g.V);  // EnergyDensity.cpp:26
                o[1] = all.y * inv4pi2;                 // TopologicalCharge.cpp:21
                *d->slot = *d->slot + 1;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------- layouts
// File order (double, [s][mu][k][re,im]) <-> device layout in precision R.
// The 32 sites of one layout block occupy one contiguous run in both orders
// (file: 32 x 36 complex, site-major; device: 36 x 32 complex, entry-major),
// so a block of CONV_THREADS threads moves one layout block as a transpose
// through shared memory: both the global read and the global write are
// consecutive 16-byte (or 8-byte) words across the warp.  Sites past V in
// the last block are neither read nor written.
constexpr int CONV_THREADS = 256;
constexpr int CONV_PITCH = 37;  // 36 entries + 1: columns of the transpose hit distinct banks

template <typename R>
__global__ void __launch_bounds__(CONV_THREADS) k_to_device(const double2* __restrict__ file, cplx<R>* __restrict__ U,
                                                            int V) {
    __shared__ double2 t[LAYOUT_BLOCK * CONV_PITCH];
    const int b = blockIdx.x;
    const int s0 = b * LAYOUT_BLOCK;
    const int ns = min(LAYOUT_BLOCK, V - s0);
    const double2* src = file + (size_t)s0 * 36;
    for (int i = threadIdx.x; i < ns * 36; i += CONV_THREADS) t[(i / 36) * CONV_PITCH + i % 36] = src[i];
    __syncthreads();
    for (int j = threadIdx.x; j < 36 * LAYOUT_BLOCK; j += CONV_THREADS) {
        const int e = j / LAYOUT_BLOCK, site = j % LAYOUT_BLOCK;
        if (site < ns) {
            const double2 v = t[site * CONV_PITCH + e];
            stc(U + link_offset<R>(e / 9, e % 9, s0 + site), cmk<R>((R)v.x, (R)v.y));
        }
    }
}
template <typename R>
__global__ void __launch_bounds__(CONV_THREADS) k_to_file(const cplx<R>* __restrict__ U, double2* __restrict__ file,
                                                          int V) {
    __shared__ double2 t[LAYOUT_BLOCK * CONV_PITCH];
    const int b = blockIdx.x;
    const int s0 = b * LAYOUT_BLOCK;
    const int ns = min(LAYOUT_BLOCK, V - s0);
    for (int j = threadIdx.x; j < 36 * LAYOUT_BLOCK; j += CONV_THREADS) {
        const int e = j / LAYOUT_BLOCK, site = j % LAYOUT_BLOCK;
        if (site < ns) {
            const cplx<R> z = ldc(U + link_offset<R>(e / 9, e % 9, s0 + site));
            t[site * CONV_PITCH + e] = make_double2((double)z.re, (double)z.im);
        }
    }
    __syncthreads();
    double2* dst = file + (size_t)s0 * 36;
    for (int i = threadIdx.x; i < ns * 36; i += CONV_THREADS) dst[i] = t[(i / 36) * CONV_PITCH + i % 36];
}

// --------------------------------------------------------- generator G
// splitmix64 finaliser (Steele, Lea & Flood, OOPSLA 2014) as a counter hash;
// h_a ~ N(0,1) by Box-Muller; U = exp(i scale sum_a h_a lambda_a/2).
__host__ __device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
__device__ __forceinline__ double unit_open(unsigned long long seed, unsigned long long ctr) {
    const unsigned long long r = mix64(seed ^ mix64(ctr));
    return ((double)(r >> 11) + 0.5) * (1.0 / 9007199254740992.0);
}

template <typename R>
__global__ void k_generate_G(cplx<R>* __restrict__ U, int V, unsigned long long seed, double scale) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * V) return;
    const int mu = t / V, s = t - mu * V;
    const unsigned long long l = (unsigned long long)s * 4ull + (unsigned long long)mu;  // file-order link index
    double h[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const unsigned long long c = l * 8ull + (unsigned long long)a;
        const double u1 = unit_open(seed, 2ull * c), u2 = unit_open(seed, 2ull * c + 1ull);
        h[a] = sqrt(-2.0 * log(u1)) * cos(6.28318530717958647692 * u2);
    }
    // X = i scale H,  H = sum_a h_a lambda_a / 2 ; coordinates of X:
    // X00 = i s (h2/2 + h7/(2 sqrt3)), X11 = i s (-h2/2 + h7/(2 sqrt3)),
    // X01 = i s (h0 - i h1)/2 = s (h1/2, h0/2), X02 = s (h4/2, h3/2), X12 = s (h6/2, h5/2)
    const double is3 = 0.57735026918962576451;
    alg<double> x;
    x.v[0] = scale * (0.5 * h[2] + 0.5 * is3 * h[7]);
    x.v[1] = scale * (-0.5 * h[2] + 0.5 * is3 * h[7]);
    x.v[2] = scale * 0.5 * h[1];
    x.v[3] = scale * 0.5 * h[0];
    x.v[4] = scale * 0.5 * h[4];
    x.v[5] = scale * 0.5 * h[3];
    x.v[6] = scale * 0.5 * h[6];
    x.v[7] = scale * 0.5 * h[5];
    const su3<double> e = expm_alg<double>(x);
    su3<R> o;
#pragma unroll
    for (int k = 0; k < 9; ++k) o.m[k] = cmk<R>((R)e.m[k].re, (R)e.m[k].im);
    store_link(U, V, mu, s, o);
}

// ------------------------------------------------------- reunitarisation
// FP32-mixed form only: rows r0, r1 by Gram-Schmidt in double, r2 = conj(r0 x r1).
template <typename R>
__global__ void k_reunitarize(cplx<R>* __restrict__ U, int V) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 4 * V) return;
    const int mu = t / V, s = t - mu * V;
    const su3<R> a = load_link(U, V, mu, s);
    cplx<double> r0[3], r1[3], r2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r0[k] = cmk<double>(a.m[k].re, a.m[k].im);
        r1[k] = cmk<double>(a.m[3 + k].re, a.m[3 + k].im);
    }
    double n0 = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) n0 += r0[k].re * r0[k].re + r0[k].im * r0[k].im;
    n0 = rsqrt(n0);
#pragma unroll
    for (int k = 0; k < 3; ++k) r0[k] = cmk<double>(r0[k].re * n0, r0[k].im * n0);
    cplx<double> d = cmk<double>(0.0, 0.0);  // <r0, r1> = sum conj(r0) r1
#pragma unroll
    for (int k = 0; k < 3; ++k) d = ccfma(r0[k], r1[k], d);
#pragma unroll
    for (int k = 0; k < 3; ++k) r1[k] = csub(r1[k], cmul(d, r0[k]));
    double n1 = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) n1 += r1[k].re * r1[k].re + r1[k].im * r1[k].im;
    n1 = rsqrt(n1);
#pragma unroll
    for (int k = 0; k < 3; ++k) r1[k] = cmk<double>(r1[k].re * n1, r1[k].im * n1);
    // r2 = conj(r0 x r1)
    r2[0] = csub(cmul(r0[1], r1[2]), cmul(r0[2], r1[1]));
    r2[1] = csub(cmul(r0[2], r1[0]), cmul(r0[0], r1[2]));
    r2[2] = csub(cmul(r0[0], r1[1]), cmul(r0[1], r1[0]));
    su3<R> o;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o.m[k] = cmk<R>((R)r0[k].re, (R)r0[k].im);
        o.m[3 + k] = cmk<R>((R)r1[k].re, (R)r1[k].im);
        o.m[6 + k] = cmk<R>((R)r2[k].re, (R)(-r2[k].im));
    }
    store_link(U, V, mu, s, o);
}

// max over links of ||U^dag U - 1||_F (x) and |det U - 1| (y), per block
template <typename R>
__global__ void __launch_bounds__(256) k_unitarity(const cplx<R>* __restrict__ U, int V, double2* __restrict__ partial) {
    __shared__ double su[256], sd[256];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double eu = 0.0, ed = 0.0;
    if (t < 4 * V) {
        const int mu = t / V, s = t - mu * V;
        const su3<R> a = load_link(U, V, mu, s);
        su3<double> b;
#pragma unroll
        for (int k = 0; k < 9; ++k) b.m[k] = cmk<double>(a.m[k].re, a.m[k].im);
        const su3<double> p = mul_an(b, b);
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const double re = p.m[k].re - ((k % 4) == 0 ? 1.0 : 0.0);
            acc += re * re + p.m[k].im * p.m[k].im;
        }
        eu = sqrt(acc);
        cplx<double> det = cmul(b.m[0], csub(cmul(b.m[4], b.m[8]), cmul(b.m[5], b.m[7])));
        det = csub(det, cmul(b.m[1], csub(cmul(b.m[3], b.m[8]), cmul(b.m[5], b.m[6]))));
        det = cadd(det, cmul(b.m[2], csub(cmul(b.m[3], b.m[7]), cmul(b.m[4], b.m[6]))));
        ed = hypot(det.re - 1.0, det.im);
    }
    su[threadIdx.x] = eu;
    sd[threadIdx.x] = ed;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            su[threadIdx.x] = fmax(su[threadIdx.x], su[threadIdx.x + w]);
            sd[threadIdx.x] = fmax(sd[threadIdx.x], sd[threadIdx.x + w]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(su[0], sd[0]);
}

// ---------------------------------------------------- per-function debug
// the plaquettes of every site and plane, as a stage's K tiles write them
template <typename R>
__global__ void k_debug_plaquettes(const cplx<R>* __restrict__ U, Geom g, R* __restrict__ K) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) plaquette_at<R>(U, K, g, s, site_coord(g, s), blockIdx.y);
}
// flow gradient Z(x, mu) for every link, file order [s][mu][9] (double2), summed as the lattice's stage form sums it
template <typename R>
__global__ void k_debug_gradient(const cplx<R>* __restrict__ U, const R* __restrict__ K, Geom g, double2* __restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x, mu = blockIdx.y;
    if (s >= g.V) return;
    const Coord c = site_coord(g, s);
    const int form = stage_form<R>(g);
    su3<R> u;
    const alg<R> Z = form == FORM_PLAQUETTE ? force_at<R>(U, K, g, s, c, mu)
                     : form == FORM_STAPLE  ? flow_gradient<R, false>(U, g, s, c, mu, u)
                                            : flow_gradient<R, true>(U, g, s, c, mu, u);
    store_alg_as_antiherm(out + ((size_t)s * 4 + mu) * 9, Z);
}

// exp(iP) for n anti-Hermitian traceless matrices given as full 3x3 (double2)
template <typename R>
__global__ void k_debug_exp(const double2* __restrict__ in, double2* __restrict__ out, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double2* m = in + (size_t)t * 9;
    alg<R> x;
    x.v[0] = (R)m[0].y;
    x.v[1] = (R)m[4].y;
    x.v[2] = (R)m[1].x;
    x.v[3] = (R)m[1].y;
    x.v[4] = (R)m[2].x;
    x.v[5] = (R)m[2].y;
    x.v[6] = (R)m[5].x;
    x.v[7] = (R)m[5].y;
    const su3<R> e = expm_alg<R>(x);
#pragma unroll
    for (int k = 0; k < 9; ++k) out[(size_t)t * 9 + k] = make_double2(e.m[k].re, e.m[k].im);
}

}  // namespace lgf
