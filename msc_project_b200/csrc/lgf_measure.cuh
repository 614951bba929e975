// E and Q of resident lattices from each Wilson loop once.
//
// The clover averages of the reference (SU3_field.cpp:533-792) sum, at every
// site and plane (mu, nu), the a x b loops of six shapes (1x1, 2x1, 3x1, 1x2,
// 1x3, 2x2) over the four quadrants around the site.  Those four loops are the
// same oriented rectangles seen from their four corners, and moving a loop's
// base point along its own border conjugates it by the links walked,
//     W(y + d) = U_d(y)^dag W(y) U_d(y),
// which commutes with the projection F[W] = -i/2 [(W - W^dag) - trace].  So a
// loop is built and projected once, at its lowest corner y,
//     H_ab(y) = c_ab F[Pn Pm^dag],  Pn = nu^b mu^a, Pm = mu^a nu^b from y,
// and its other three corners follow from the 8 real coordinates of H by
// covariant shifts (T_d H)(x) = U_d(x-d)^dag H(x-d) U_d(x-d):
//     sum of shape (a, b) at x = (1 + T_mu^a)(1 + T_nu^b) H_ab (x).
// The shifts of all shapes are nested (Horner), so a site and plane takes 16
// path products, 6 projections and 11 shifts instead of the 48 products and
// 24 projections of building every quadrant's loops at every site: 3600
// against 6900 operations.
//
//   k_meas_loops<R, ROUND>    H_ab of three planes for every site
//   k_meas_planes<R, ROUND>   shifts along nu (from memory), then along mu
//                             (through shared memory): F, F^, e and q terms
//   k_meas_sites<R>           e(x), q(x) and their sums per 32-site chunk
//   k_reduce (lgf_kernels.cuh)
//
// A round handles three planes: round 0 (01), (02), (03), round 1 their
// complements (23), (13), (12), whose q terms pair with round 0's F^.  The
// intermediates need no memory of their own: between RK3 steps the ring
// buffers U1, U2 and the accumulator A are dead (stage 1 overwrites U1 and A,
// stage 2 U2), and per 32-site block U1..U2 hold exactly 18 fields of 8 reals
// (6 shapes x 3 planes) and A four: F^ of round 0's planes, and the e terms.
//
// One B200, whole measurement without the reduction, against one kernel that
// builds every quadrant's loops at every site: FP64 16^4 0.357 -> 0.21 ms,
// 24^3x48 3.58 -> 1.75 ms, 48^4 28.8 -> 14.3 ms; FP32-mixed 24^3x48 2.28 ->
// 1.22 ms, 48^4 18.5 -> 9.5 ms.  24^3x48 FP64 in parts: loops 0.43 + 0.41 ms
// (FP64 pipe 58-62% busy, then L2 latency), planes 0.44 + 0.43 ms (1.3 KB read
// per site and plane: 0.31 ms with every load in L1, 0.38 without arithmetic).
#pragma once
#include "lgf_kernels.cuh"

namespace lgf {

constexpr int LOOP_SHAPES = 6;                     // (1,1) (2,1) (3,1) (1,2) (1,3) (2,2)
constexpr int LOOP_FIELDS = 3 * LOOP_SHAPES;       // of one round
static_assert(LOOP_FIELDS * FIELD_REALS == 2 * 36 * 2 * LAYOUT_BLOCK, "U1..U2 hold one round's fields");

// planes of a round, and the shapes' weights in F^ (F = G / 4, F^ = 19/36 G +
// the weighted sum of the others; G the unweighted 1x1 sum)
template <int ROUND> __host__ __device__ __forceinline__ int round_mu(int j) { return ROUND == 0 ? 0 : (j == 0 ? 2 : 1); }
template <int ROUND> __host__ __device__ __forceinline__ int round_nu(int j) { return ROUND == 0 ? j + 1 : (j == 2 ? 2 : 3); }

// field f (0..17) of site s in the round's scratch, a pointer to its first
// vector: 8 coordinates as double2 pairs or float4 quads, planes of 32 sites
template <typename R> __device__ __forceinline__ R* loop_field(R* W, int f, int s) {
    return W + ((size_t)(s / LAYOUT_BLOCK) * LOOP_FIELDS + f) * FIELD_REALS + (s % LAYOUT_BLOCK) * (16 / sizeof(R));
}
// the same in the accumulator's layout (four fields per block)
template <typename R> __device__ __forceinline__ R* acc_field(R* A, int f, int s) {
    return A + ((size_t)(s / LAYOUT_BLOCK) * 4 + f) * FIELD_REALS + (s % LAYOUT_BLOCK) * (16 / sizeof(R));
}
// ------------------------------------------------------------------- loops
// H_ab of the round's three planes: one thread per site and plane, warp w of
// a block takes plane w % 3 of tile group w / 3 (a tile = 32 sites; adjacent
// tiles share a block, so their links meet in its L1).  No barriers.  A path
// that is extended again later keeps its first two rows in the thread's own
// shared-memory column: the products rebuild the third row, and the column
// keeps the peak of live registers at three matrices.
constexpr int LOOP_MAX_GROUPS = 4;
constexpr int LOOP_STASH = 3;  // parked paths per thread
// The loops of FP32 links are multiplied and projected in double too: one
// loop's error now enters the sums at four sites, and on a flowed field the
// projection is small against the paths' unit-size entries.  In float the
// charge of a flowed 6x10x14x18 lattice was off by 7.5e-6 of itself against
// 2.5e-6 with every quadrant's loops built apart.  H and its shifts stay float.
typedef double LoopReal;

// Lattices of up to one 32-site tile per SM are measured by the one-launch
// kernel k_measure instead (lgf_kernels.cuh): with too few threads to fill the
// SMs its 33 us (FP64, 8^4) beat the five launches' 46 us.  Above, the SMs with
// two tiles run them in turn: FP64 4800 to 8192 sites 61 against 47 us, 10000
// 86 against 63, 12^4 138 against 105; FP32, whose loops are multiplied in
// double here, 41 to 42 against 43 to 45, 10000 57 against 54, 12^4 88 against 84.  The rule reads the lattice alone,
// so a lattice gives the same bits in every group.
constexpr int SMALL_MEAS_TILES = 148;
__host__ __device__ __forceinline__ bool small_measure(const Geom& g) {
    return (long long)g.n[0] * ((g.Vs + MEAS_SITES - 1) / MEAS_SITES) <= SMALL_MEAS_TILES;
}

template <typename R> struct LoopStash {
    typename vec2_of<R>::type* p;  // entry k at p[k * stride]
    int stride;
    __device__ __forceinline__ void put(const su3<R>& P) const {
#pragma unroll
        for (int k = 0; k < MEAS_STASH_ENTRIES; ++k) {
            typename vec2_of<R>::type v;
            v.x = P.m[k].re;
            v.y = P.m[k].im;
            p[k * stride] = v;
        }
    }
    __device__ __forceinline__ su3<R> get() const {
        su3<R> P;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            if (k < MEAS_STASH_ENTRIES) {
                const typename vec2_of<R>::type v = p[k * stride];
                P.m[k] = cmk<R>(v.x, v.y);
            } else {
                P.m[k] = cmk<R>(R(0), R(0));  // never read: the next product rebuilds the row
            }
        }
        return P;
    }
};

inline size_t loops_smem_bytes(int groups) {
    return (size_t)LOOP_STASH * MEAS_STASH_ENTRIES * sizeof(double2) * 96 * groups;
}

template <typename R, int ROUND>
__global__ void __launch_bounds__(96 * LOOP_MAX_GROUPS, 1) k_meas_loops(const LatDesc<R>* __restrict__ descs,
                                                                         const int4* __restrict__ mtiles,
                                                                         const int2* __restrict__ seg) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x, j = threadIdx.y % 3, grp = threadIdx.y / 3, groups = blockDim.y / 3;
    const int nthr = MEAS_SITES * blockDim.y, column = threadIdx.y * MEAS_SITES + lane;
    typedef LoopReal D;
    typedef typename vec2_of<D>::type V2;
    V2* st = reinterpret_cast<V2*>(smem_raw) + column;
    const LoopStash<D> sa{st, nthr}, sb{st + MEAS_STASH_ENTRIES * nthr, nthr}, sl{st + 2 * MEAS_STASH_ENTRIES * nthr, nthr};
    const int mu = round_mu<ROUND>(j), nu = round_nu<ROUND>(j);
    const D k12 = -4.0 / 45.0, k13 = 1.0 / 120.0, k22 = 1.0 / 144.0;
    const int2 r = *seg;  // this launch's tiles: mtiles[r.x, r.x + r.y)
    for (int ti = r.x + blockIdx.x * groups + grp; ti < r.x + r.y; ti += gridDim.x * groups) {
        const int4 tile = mtiles[ti];
        const LatDesc<R>* d = descs + tile.x;
        const Geom g = d->g;
        const int off = meas_site_offset(tile.z, lane);
        if (off >= g.Vs) continue;
        const int s = tile.y * g.Vs + off;
        const Coord c = site_coord(g, s);
        Plane<R, D> P;
        P.U = d->U0;
        P.V = g.V;
        P.mu = mu;
        P.nu = nu;
        P.dm = dir_of(g, c, mu);
        P.dn = dir_of(g, c, nu);
        R* W = loop_field<R>(reinterpret_cast<R*>(d->U1), j * LOOP_SHAPES, s);
        const PlanePos x0 = {s, P.dm.x, P.dn.x};
        // (1,1)
        PlanePos pn = x0;
        su3<D> Pn = P.step(pn, false, 1);
        P.ext(Pn, pn, true, 1);  // Pn(1,1)
        PlanePos pm = x0;
        su3<D> Pm = P.step(pm, true, 1);
        P.ext(Pm, pm, false, 1);  // Pm(1,1)
        put_field(W, leaf<R>(Pn, Pm, D(1)));
        sa.put(Pm);
        // (2,1)
        P.ext(Pn, pn, true, 1);  // Pn(2,1)
        PlanePos pl = x0;
        Pm = P.step(pl, true, 1);
        P.ext(Pm, pl, true, 1);  // mu^2
        sl.put(Pm);
        PlanePos p21 = pl;
        P.ext(Pm, p21, false, 1);  // Pm(2,1)
        put_field(W + FIELD_REALS, leaf<R>(Pn, Pm, k12));
        sb.put(Pm);
        // (3,1)
        P.ext(Pn, pn, true, 1);  // Pn(3,1)
        Pm = sl.get();
        P.ext(Pm, pl, true, 1);  // mu^3
        P.ext(Pm, pl, false, 1);  // Pm(3,1)
        put_field(W + 2 * FIELD_REALS, leaf<R>(Pn, Pm, k13));
        // (1,2)
        Pm = sa.get();
        P.ext(Pm, pm, false, 1);  // Pm(1,2)
        pl = x0;
        Pn = P.step(pl, false, 1);
        P.ext(Pn, pl, false, 1);  // nu^2
        sl.put(Pn);
        PlanePos p12 = pl;
        P.ext(Pn, p12, true, 1);  // Pn(1,2)
        put_field(W + 3 * FIELD_REALS, leaf<R>(Pn, Pm, k12));
        sa.put(Pn);
        // (1,3)
        P.ext(Pm, pm, false, 1);  // Pm(1,3)
        Pn = sl.get();
        P.ext(Pn, pl, false, 1);  // nu^3
        P.ext(Pn, pl, true, 1);   // Pn(1,3)
        put_field(W + 4 * FIELD_REALS, leaf<R>(Pn, Pm, k13));
        // (2,2)
        Pn = sa.get();
        P.ext(Pn, p12, true, 1);  // Pn(2,2)
        Pm = sb.get();
        P.ext(Pm, p21, false, 1);  // Pm(2,2)
        put_field(W + 5 * FIELD_REALS, leaf<R>(Pn, Pm, k22));
    }
}

// ------------------------------------------------------------------ planes
// A unit of k_meas_planes is a block of columns along mu of one plane: C
// columns (adjacent sites: the runs a warp reads) times every x_mu, so that
// the shifts along mu stay inside the unit.  Extents above the unit's size
// are cut into row tiles that recompute the three rows before them.
struct ColumnTiling {
    int C;       // columns of a unit
    int rows;    // rows of a unit: the extent, or the whole unit (with 3 rows of halo)
    int tiles;   // row tiles per column block
    int ncol;    // columns of the lattice along mu
    int blocks;  // column blocks
    __host__ __device__ __forceinline__ bool cyclic() const { return tiles == 1; }
    __host__ __device__ __forceinline__ int units() const { return blocks * tiles; }
};
__host__ __device__ __forceinline__ ColumnTiling column_tiling(const Geom& g, int mu, int unit_sites) {
    ColumnTiling t;
    const int n = sel4(mu, g.n[0], g.n[1], g.n[2], g.n[3]);
    t.ncol = g.V / n;
    if (n <= unit_sites) {
        t.C = unit_sites / n;
        if (t.C > 1) t.C &= ~1;  // whole 32-byte sectors
        t.rows = n;
        t.tiles = 1;
    } else {
        t.C = 1;
        t.rows = unit_sites;
        t.tiles = (n + unit_sites - 4) / (unit_sites - 3);
    }
    t.blocks = (t.ncol + t.C - 1) / t.C;
    return t;
}
// units of a lattice in one round
__host__ __device__ __forceinline__ int plane_units(const Geom& g, int round, int unit_sites) {
    if (round == 0) return 3 * column_tiling(g, 0, unit_sites).units();
    return column_tiling(g, 2, unit_sites).units() + 2 * column_tiling(g, 1, unit_sites).units();
}
struct PlaneUnit {
    int j;      // plane of the round
    int block;  // column block
    int tile;   // row tile
};
// unit u of a lattice; round 0's planes share mu = 0 and are interleaved
template <int ROUND> __host__ __device__ __forceinline__ PlaneUnit plane_unit(const Geom& g, int unit_sites, int u) {
    PlaneUnit p;
    int v;
    if (ROUND == 0) {
        p.j = u % 3;
        v = u / 3;
    } else {
        const int n2 = column_tiling(g, 2, unit_sites).units();
        p.j = u < n2 ? 0 : 1 + (u - n2) % 2;
        v = u < n2 ? u : (u - n2) / 2;
    }
    const int tiles = column_tiling(g, round_mu<ROUND>(p.j), unit_sites).tiles;
    p.block = v / tiles;
    p.tile = v % tiles;
    return p;
}
// site of (column, row) of a unit: row 0 of a halo tile lies 3 rows before its first output
struct UnitSite { int s, xmu, out; };
__host__ __device__ __forceinline__ bool unit_site(const Geom& g, int mu, const ColumnTiling& t, const PlaneUnit& p, int col,
                                                   int row, UnitSite* o) {
    const int n = sel4(mu, g.n[0], g.n[1], g.n[2], g.n[3]), stride = sel4(mu, g.stride[0], g.stride[1], g.stride[2], g.stride[3]);
    const int c = p.block * t.C + col;
    if (c >= t.ncol || row >= t.rows) return false;
    int x = row;
    o->out = 1;
    if (!t.cyclic()) {
        const int first = p.tile * (t.rows - 3);
        o->out = row >= 3 && first + row - 3 < n;
        x = (first + row - 3 + n) % n;
    }
    const int outer = c / stride, inner = c - outer * stride;
    o->xmu = x;
    o->s = (outer * n + x) * stride + inner;
    return true;
}

// Table of the members a launch measures, in list order: units of member k
// are [start, next start).
struct PlaneMember { int member, start; };

template <typename R> inline size_t planes_smem_bytes(int unit_sites) { return (size_t)4 * 8 * sizeof(R) * unit_sites; }

template <typename R> struct UnitField {  // a shift's input at every site of the unit
    R* p;
    int n;
    __device__ __forceinline__ void put(int t, const alg<R>& z) const {
        typedef typename vec2_of<R>::type V2;
        V2* v = reinterpret_cast<V2*>(p);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            V2 w;
            w.x = z.v[2 * k];
            w.y = z.v[2 * k + 1];
            v[k * n + t] = w;
        }
    }
    __device__ __forceinline__ alg<R> get(int t) const {
        typedef typename vec2_of<R>::type V2;
        const V2* v = reinterpret_cast<const V2*>(p);
        alg<R> z;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const V2 w = v[k * n + t];
            z.v[2 * k] = w.x;
            z.v[2 * k + 1] = w.y;
        }
        return z;
    }
};

// Sites of a unit (threads of a block) and resident blocks per SM: the more
// columns, the longer the runs a warp reads (4 columns of 48 rows instead of
// 8: 24^3x48 9% and 48^4 20% slower), so FP64 takes one block of 384 at 168
// registers; float fits two at 80 (947 against 1026 us for all five kernels
// on 24^3x48, 7.9 against 8.3 ms on 48^4 with one block at 160).
constexpr int PLANE_MAX_SITES = 384;
template <typename R> constexpr int plane_blocks() { return sizeof(R) == sizeof(double) ? 1 : 2; }

template <typename R, int ROUND, bool OUT>
__global__ void __launch_bounds__(PLANE_MAX_SITES, plane_blocks<R>()) k_meas_planes(const LatDesc<R>* __restrict__ descs,
                                                                     const PlaneMember* __restrict__ members,
                                                                     const int* __restrict__ nmembers,
                                                                     const int2* __restrict__ seg, MeasSites out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int T = blockDim.x, t = threadIdx.x;
    R* sm = reinterpret_cast<R*>(smem_raw);
    const UnitField<R> fg{sm, T}, f1{sm + 8 * T, T}, f2{sm + 16 * T, T}, f3{sm + 24 * T, T};
    const int2 r = *seg;  // this launch's units
    const int nm = *nmembers;
    for (int u = r.x + blockIdx.x; u < r.x + r.y; u += gridDim.x) {
        int lo = 0, hi = nm;  // the member whose units hold u
        while (hi - lo > 1) {
            const int mid = (lo + hi) / 2;
            if (members[mid].start <= u) lo = mid; else hi = mid;
        }
        const LatDesc<R>* d = descs + members[lo].member;
        const Geom g = d->g;
        const PlaneUnit pu = plane_unit<ROUND>(g, T, u - members[lo].start);
        const int j = pu.j, mu = round_mu<ROUND>(j), nu = round_nu<ROUND>(j);
        const ColumnTiling ct = column_tiling(g, mu, T);
        const int row = t / ct.C, col = t - row * ct.C;
        UnitSite us;
        const bool in = unit_site(g, mu, ct, pu, col, row, &us);
        const cplx<R>* __restrict__ U = d->U0;
        const R* W = reinterpret_cast<const R*>(d->U1);
        alg<R> G, F;  // own terms: (1 + T_nu) of 1x1; the weighted sums of the other shapes
        if (in) {
            const int s = us.s;
            const int nn = sel4(nu, g.n[0], g.n[1], g.n[2], g.n[3]), sn = sel4(nu, g.stride[0], g.stride[1], g.stride[2], g.stride[3]);
            const int xn = (int)(((unsigned)s / (unsigned)sn) % (unsigned)nn);
            const int s1 = xn >= 1 ? s - sn : s + (nn - 1) * sn;
            const int s2 = xn >= 2 ? s - 2 * sn : s + (nn - 2) * sn;
            const int s3 = xn >= 3 ? s - 3 * sn : s + (nn - 3) * sn;
            const int f0 = j * LOOP_SHAPES;
            auto H = [&](int f, int q) { return get_field<R, true>(loop_field(W, f0 + f, q)); };
            // each load is issued one or two shifts ahead of its use (loads beside
            // their shifts: 500 + 459 us on 24^3x48 FP64 instead of 440 + 428)
            const su3<R> l3 = load_link(U, g.V, nu, s3);
            alg<R> a = H(4, s3);  // (1,3) at x - 3nu
            const su3<R> l2 = load_link(U, g.V, nu, s2);
            const alg<R> h3 = H(3, s2);  // (1,2) at x - 2nu
            alg<R> b = H(5, s2);  // (2,2) at x - 2nu
            a = shift(a, l3);
            const su3<R> l1 = load_link(U, g.V, nu, s1);
            const alg<R> h30 = H(3, s);
            const alg<R> h40 = H(4, s);
            a = shift(alg_add(h3, a), l2);
            const alg<R> h11 = H(1, s1);  // (2,1) at x - nu
            b = shift(b, l2);
            const alg<R> h10 = H(1, s), h50 = H(5, s);
            a = shift(a, l1);
            F = alg_add(alg_add(h30, h40), a);
            f1.put(t, F);
            const alg<R> h21 = H(2, s1), h20 = H(2, s);  // (3,1)
            a = shift(alg_add(h11, b), l1);
            a = alg_add(alg_add(h10, h50), a);
            f2.put(t, a);
            F = alg_add(F, a);
            const alg<R> h01 = H(0, s1), h00 = H(0, s);  // (1,1)
            a = alg_add(h20, shift(h21, l1));
            f3.put(t, a);
            F = alg_add(F, a);
            G = alg_add(h00, shift(h01, l1));
            fg.put(t, G);
        }
        __syncthreads();
        if (in && us.out) {
            const int s = us.s, n = sel4(mu, g.n[0], g.n[1], g.n[2], g.n[3]), sd = sel4(mu, g.stride[0], g.stride[1], g.stride[2], g.stride[3]);
            const int x = us.xmu, all = ct.rows * ct.C;
            const int s1 = x >= 1 ? s - sd : s + (n - 1) * sd;
            const int s2 = x >= 2 ? s - 2 * sd : s + (n - 2) * sd;
            const int s3 = x >= 3 ? s - 3 * sd : s + (n - 3) * sd;
            const int t1 = t - ct.C < 0 ? t - ct.C + all : t - ct.C;  // (a halo tile's outputs never wrap)
            const int t2 = t1 - ct.C < 0 ? t1 - ct.C + all : t1 - ct.C;
            const int t3 = t2 - ct.C < 0 ? t2 - ct.C + all : t2 - ct.C;
            su3<R> l = load_link(U, g.V, mu, s3);
            alg<R> a = shift(f3.get(t3), l);
            l = load_link(U, g.V, mu, s2);
            a = shift(alg_add(f2.get(t2), a), l);
            l = load_link(U, g.V, mu, s1);
            F = alg_add(F, shift(alg_add(f1.get(t1), a), l));
            G = alg_add(G, shift(fg.get(t1), l));
            alg<R> F11;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                F11.v[k] = R(0.25) * G.v[k];
                F.v[k] = fma(R(19.0 / 36.0), G.v[k], F.v[k]);  // F^
            }
            if (OUT) {
                const int p = ROUND == 0 ? j : 5 - j;
                if (out.dbg_clover) store_alg_as_herm(out.dbg_clover + ((size_t)s * 6 + p) * 9, F11);
                if (out.dbg_improved) store_alg_as_herm(out.dbg_improved + ((size_t)s * 6 + p) * 9, F);
                if (out.swap) {
                    const alg<R> z = F;
                    F = F11;
                    F11 = z;
                }
            }
            const double e = retr_hh(F11, F11);
            R* slot = acc_field(d->A, j, s);
            if (ROUND == 0) {
                put_field(slot, F);
                reinterpret_cast<double*>(acc_field(d->A, 3, s - s % LAYOUT_BLOCK))[j * LAYOUT_BLOCK + s % LAYOUT_BLOCK] = e;
            } else {
                // the complementary plane's F^; its slot then takes this plane's e and q terms
                const double q = retr_hh(F, get_field<R, false>(slot));
                *reinterpret_cast<double2*>(slot) = make_double2(e, q);
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------- sites
// e(x), q(x) from the planes' terms and their sums per 32-site chunk: warp w
// of a block takes one tile.
//   e(x) = sum_{mu<nu} ReTr(F F)                 (EnergyDensity.cpp:13-20)
//   q(x) = ReTr(F^32 F^01) + ReTr(F^31 F^20) + ReTr(F^30 F^12)
//        = -T(23,01) + T(13,02) - T(03,12),  T(a,b) = ReTr(F^a F^b)
//                                             (TopologicalCharge.cpp:11-16)
constexpr int SITES_THREADS = 256;

template <typename R, bool OUT>
__global__ void __launch_bounds__(SITES_THREADS) k_meas_sites(const LatDesc<R>* __restrict__ descs,
                                                             const int4* __restrict__ mtiles,
                                                             const int2* __restrict__ seg, MeasSites out) {
    const int lane = threadIdx.x & 31, warps = SITES_THREADS / 32;
    const int2 r = *seg;
    for (int ti = r.x + blockIdx.x * warps + (threadIdx.x >> 5); ti < r.x + r.y; ti += gridDim.x * warps) {
        const int4 tile = mtiles[ti];
        const LatDesc<R>* d = descs + tile.x;
        const Geom g = d->g;
        const int off = meas_site_offset(tile.z, lane);
        double e = 0.0, q = 0.0;
        if (off < g.Vs) {
            const int s = tile.y * g.Vs + off;
            const double* e0 = reinterpret_cast<const double*>(acc_field(d->A, 3, s - s % LAYOUT_BLOCK)) + s % LAYOUT_BLOCK;
            const double2 v0 = *reinterpret_cast<const double2*>(acc_field(d->A, 0, s));  // plane 23
            const double2 v1 = *reinterpret_cast<const double2*>(acc_field(d->A, 1, s));  // plane 13
            const double2 v2 = *reinterpret_cast<const double2*>(acc_field(d->A, 2, s));  // plane 12
            e = ((e0[0] + e0[LAYOUT_BLOCK]) + (e0[2 * LAYOUT_BLOCK] + v2.x)) + (v1.x + v0.x);
            q = -v0.y + v1.y - v2.y;
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
        if (lane == 0) d->partial[tile.y * d->nchunk + tile.z] = make_double2(e, q);
    }
}

}  // namespace lgf
