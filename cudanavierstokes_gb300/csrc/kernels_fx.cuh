// kernels_fx.cuh -- FP64 mode: fixed-point stencil inputs, dilatation and the RHS of one
// point (fx.cuh explains the number format).
//
// Per stage, from the ghosted FP64 fields and their ranges:
//   fx_column   the eight fields of a column of points as integers, and theta from the
//               integers of u, v, w (fx_point: of one point)
//   fx_ghost    the same conversion of a ghost cell
//   fx_table    the stage's scale factors (one thread each)
//   fx_convective, fx_viscous  the two parts of the RHS of a point on the integer units; each
//               sum is converted once
// Where the fields' ranges are too wide for their common exponents (fx_exponents) the stage takes
// theta from wide_theta and the RHS from rhs_wide, FP64 sums of the FP64 fields.
#pragma once
#include "cns_common.cuh"
#include "cns_internal.h"
#include "fx.cuh"
#include "kernels_point.cuh"

namespace cns {

// Exponents of the eight fields from their ranges; false: the stage takes FP64 sums. A value is
// held to 2^-62 of its field's maximum, so the sums serve
//   fields within 2^-300 .. 2^300 (fx_valid);
//   rho and T that vary by at most FX_SPAN binades over the box, ghosts included (a ratio of 8 to
//   16), T by less where mu's exponent is large: each value of rho, T, p, mu is then held exactly,
//   and the sums' units, which come from the maxima, are near every point's own (T 1 to 10: a
//   point's error is up to 5e-15 of the largest value near it, T 1 to 1e3: 7e-13, FP64 1e-15);
//   rho |u|^2 < 2^8 p: what velocities lose in a region at rest stays below the rounding of its
//   pressure.
__device__ __forceinline__ bool fx_exponents(const FxBase& b, const unsigned* slots, int (&e)[8]) {
    unsigned m[8];
    fx_slots(slots, m);
    const uint2 least = __ldcg((const uint2*)(slots + FX_LEAST));
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        e[q] = fx_exponent(m[q]);
        ok = ok && fx_valid(m[q]);
    }
    // binades from the smallest magnitude's to the largest's
    const int sr = (int)(m[0] + least.x) - 2048, st = (int)(m[4] + least.y) - 2048;
    return ok && sr <= FX_SPAN && st <= b.span_T && e[0] + 2 * max(e[1], max(e[2], e[3])) <= e[5] - sr - st + 8;
}

// Units. Each sum of the RHS that joins several integer sums has a unit U of its own: the
// factor K of a term becomes the integer K / U 2^64 <= 2^63 (1 - 2^-20) (equal for the largest
// K of the sum) and fx_mul of the two gives the term. The gradients and theta have a power of
// two, 2^G, with factors below 2^62. So every sum is kept to 2^-59 or finer of the largest
// value that its terms can take; the conversion to FP64 is relative to the value itself.
constexpr double FX_FULL = 0x1p63 * (1.0 - 0x1p-20);

// x 2^n of a positive normal number on the integer units, kept within the normal range
__device__ __forceinline__ double fx_scaled(double x, int n) {
    const int hi = __double2hiint(x);
    const int ex = min(max((hi >> 20) + n, 1), 2046);
    return __hiloint2double((ex << 20) | (hi & 0xfffff), __double2loint(x));
}
__device__ __forceinline__ double fx_larger(double x, double y) {   // of positive numbers
    const i64 a = __double_as_longlong(x), b = __double_as_longlong(y);
    return a > b ? x : y;
}
__device__ __forceinline__ int fx_log2(double x) { return (__double2hiint(x) >> 20) - 1023; }   // floor

// unit of theta, 2^x: the largest of its three factors in [2^61, 2^62), theta < 2^61.4
__device__ __forceinline__ int fx_unit_theta(const FxBase& b, const int (&e)[8]) {
    return fx_log2(fx_larger(fx_scaled(b.thmax, e[1] - 62),
                             fx_larger(fx_scaled(b.th[1], e[2] - 62), fx_scaled(b.th[2], e[3] - 62)))) + 3;
}

// the factors of theta = sum_d (weighted difference of the d-th velocity)_d k_d; xp: 1/x' of
// the point on a stretched x
__device__ __forceinline__ void fx_theta_factors(const FxBase& b, const int (&e)[8], int nonuniform_x, double xp,
                                                 i64& kx, i64& ky, i64& kz) {
    const int n = fx_unit_theta(b, e);   // K 2^(64 - n) = (K 2^(62 - m)) with m = n - 2
    kx = fx_from(fx_scaled(nonuniform_x ? b.th[0] * xp : b.th[0], e[1] - 62), n - 2);
    ky = fx_from(fx_scaled(b.th[1], e[2] - 62), n - 2);
    kz = fx_from(fx_scaled(b.th[2], e[3] - 62), n - 2);
}

// the factor of sum q (FXK_*) in direction d; xth: the exponent of theta's unit. Mass flux: Q
// in units of 2^(e_rho + e_g - 60), weight 1/2; cubic fluxes: Q phi in units of 2^(e_rho + e_g
// + e_phi - 58), doubled, weight 1/4. On a stretched x the first derivatives' sums are
// multiplied by x'^-1 / xpmax 2^63 (1 - 2^-20) / 2^64 beforehand (in the base factors).
__device__ __forceinline__ double fx_factor(const FxBase& b, const int (&e)[8], int xth, int d, int q) {
    const auto pick = [&](const double (&a)[3]) { return d == 0 ? a[0] : d == 1 ? a[1] : a[2]; };
    const auto ev = [&](int n) { return n == 0 ? e[1] : n == 1 ? e[2] : e[3]; };   // u, v, w
    if (q < FXK_MU) return fx_scaled(pick(b.b1V), ev(q) - 62);
    if (q == FXK_MU) return fx_scaled(pick(b.b1V), e[7] - 62);
    if (q == FXK_T) return fx_scaled(pick(b.b1V), e[4] - 62);
    if (q == FXK_TH) return fx_scaled(pick(b.b1V3), xth);
    if (q == FXK_P) return fx_scaled(pick(b.b1S), e[5] - 62);
    if (q < FXK_LT) return fx_scaled(pick(b.b2), ev(q - FXK_L) - 62);
    if (q == FXK_LT) return fx_scaled(pick(b.b2), e[4] - 62);
    const int er = e[0] + ev(d);
    if (q == FXK_F0) return fx_scaled(pick(b.b1S), er - 61);
    return fx_scaled(pick(b.b1S), er + (q == FXK_F + 3 ? e[6] : ev(q - FXK_F)) - 61);
}

// entry t of the stage's table (FXK_*)
static __device__ __noinline__ i64 fx_table(const FxBase& b, const unsigned* gmax, double lam_mu, int t) {
    int e[8];
    const bool wide = !fx_exponents(b, gmax, e);
    if (wide || t == FXK_WIDE) return wide;
    const int xth = fx_unit_theta(b, e);
    const auto K = [&](int d, int q) { return fx_factor(b, e, xth, d, q); };
    const auto ev = [&](int q) { return q == 1 ? e[1] : q == 2 ? e[2] : q == 3 ? e[3] : e[6]; };   // u, v, w, H
    const auto big = [&](int q) { return fx_larger(K(0, q), fx_larger(K(1, q), K(2, q))); };
    // units (2^64 / FX_FULL of the largest factor): the gradients' power of two, above 4 times
    // their largest factor; the mass sum; the fluxes of equation q with its centre term's factor;
    // second derivatives of component q
    const int xg = fx_log2(fx_larger(big(FXK_U), fx_larger(big(FXK_U + 1), big(FXK_U + 2)))) + 3;
    const double U0 = big(FXK_F0) * (0x1p64 / FX_FULL);
    const auto ctr = [&](int q) { return fx_scaled(U0, ev(q) - 1); };
    const auto UA = [&](int q) {
        if (q == 0) return U0;
        return fx_larger(big(FXK_F0 + q), ctr(q)) * (0x1p64 / FX_FULL);
    };
    const auto UL = [&](int q) { return big(FXK_L + q) * (0x1p64 / FX_FULL); };
    const double UM = big(FXK_MU) * (0x1p64 / FX_FULL), UT = big(FXK_T) * (0x1p64 / FX_FULL);
    const auto factor = [&](double k, double unit) {   // low word, balanced high half
        const i64 v = __double2ll_rn(k / unit * 0x1p64);
        return (i64)(((unsigned long long)(unsigned)fx_hi(v) << 32) | (unsigned)fx_lo(v));
    };
    if (t < 3 * FXK_DIR) {
        const int d = t / FXK_DIR, q = t % FXK_DIR;
        if (q == FXK_P) return __double_as_longlong(K(d, q));
        if (q == FXK_TH) return __double_as_longlong(fx_scaled(K(d, q), e[7] + 2));   // with mu
        const double u = q < FXK_MU ? fx_pow2(xg) : q == FXK_MU ? UM : q == FXK_T ? UT
                         : q <= FXK_LT ? UL(q - FXK_L) : UA(q - FXK_F0);
        return factor(K(d, q), u);
    }
    if (t == FXK_TG) return factor(fx_scaled(1.0 / 3.0, xth), fx_pow2(xg));
    if (t < FXK_A) return factor(ctr(1 + t - FXK_CTR), UA(1 + t - FXK_CTR));
    // units as doubles: the five sums; mu times the second derivatives (of T: with lambda/mu);
    // stress . grad mu, grad T . grad mu (with lambda/mu), the dissipation
    const double um = fx_pow2(e[7] + 2);
    return __double_as_longlong(t < FXK_UL ? UA(t - FXK_A) : t < FXK_UL + 3 ? um * UL(t - FXK_UL)
                                : t == FXK_UL + 3 ? lam_mu * um * UL(3) : t == FXK_UD ? fx_pow2(xg + 64) * UM
                                : t == FXK_UC ? lam_mu * 0x1p64 * UT * UM : fx_pow2(2 * xg + 64));
}

// a0 b0 + a1 b1, / 2^62: the second derivative on a stretched x, 1/x'^2 f'' - x''/x'^3 f' of
// the index derivatives' sums b0 < 2^61, b1 < 2^61.8 with |a0| / 2 + 0.87 |a1| <= 2^62 (1 -
// 2^-19): the cross sum < 2^62.9, the value < 2^62
__device__ __forceinline__ i64 fx_mul2(i64 a0, i64 b0, i64 a1, i64 b1) {
    const int a0h = fx_hi(a0), a0l = fx_lo(a0), a1h = fx_hi(a1), a1l = fx_lo(a1);
    const int b0h = fx_hi(b0), b0l = fx_lo(b0), b1h = fx_hi(b1), b1l = fx_lo(b1);
    const i64 m = fx_mad(a0h, b0l, fx_mad(a0l, b0h, fx_mad(a1h, b1l, fx_mad(a1l, b1h, FX_HALF / 4))));
    return (fx_mad(a0h, b0h, fx_mad(a1h, b1h, 0)) << 2) + (m >> 30);
}

// the eight fields of element c as integers, the velocities given
__device__ __forceinline__ void fx_store(const FxFields& o, const int (&e)[8], int c, i64 u, i64 v, i64 w,
                                         const double (&q)[5]) {   // q: rho, T, p, H, mu
    fx_store4(o.v + c, u, v, w, fx_from(q[2], e[5]));
    o.t[c] = make_longlong2(fx_from(q[1], e[4]), fx_from(q[4], e[7]));
    o.r[c] = make_longlong2(fx_from(q[0], e[0]), fx_from(q[3], e[6]));
}
// rho, T, p, H, mu of element c
__device__ __forceinline__ void fx_scan(const RhsIn<double>& in, int c, double (&q)[5]) {
    q[0] = in.r[c]; q[1] = in.t[c]; q[2] = in.p[c]; q[3] = in.h[c]; q[4] = in.m[c];
}

// the conversion of ghost cell t (wide: its ranges alone)
__device__ __forceinline__ void fx_ghost(const Geom& g, const RhsIn<double>& in, const int (&e)[8], int t, bool wide,
                                         FxLeast& least) {
    const GhostCell gc = ghost_cell_of(g, t);
    const int off = gc.side == 0 ? -gc.m : gc.m - 1;
    const int c = (int)(gc.face == 0   ? g.at(gc.side == 0 ? off : g.mx + off, gc.j, gc.k)
                        : gc.face == 1 ? g.at(gc.i, gc.side == 0 ? off : g.my + off, gc.k)
                                       : g.at(gc.i, gc.j, gc.side == 0 ? off : g.mz + off));
    double q[5];
    fx_scan(in, c, q);
    least.add(q[0], q[1]);
    if (!wide) fx_store(in.fx, e, c, fx_from(in.u[c], e[1]), fx_from(in.v[c], e[2]), fx_from(in.w[c], e[3]), q);
}

// Conversion of a column of points and its theta. The threads (tx, ty), tx < 32, ty < TY, own
// the x-y tile at (i0, j0) and march the planes [k0, k1): u of the tile rows with V halo
// points on either side and v of the tile columns in shared memory, w of the planes k - V ..
// k + V in a register ring, so that a point converts ~9.4 values instead of the 8 + 6V of
// fx_point (a conversion is ~20 instructions: 8.6 against 32 made the kernel ALU bound); the
// next plane's loads are issued before the current plane is computed. Tile slots beyond [-V,
// mx + V) x [-V, my + V) are read by no interior point and not loaded. All threads of the
// block call it.
template <int V, int TY>
__device__ __forceinline__ void fx_column(const Geom& g, const FxBase& b, const RhsIn<double>& in, const int (&e)[8],
                                          const double* __restrict__ xp, int i0, int j0, int k0, int k1, bool own,
                                          int tx, int ty, i64 (*su)[32 + 2 * V], i64 (*sv)[32], FxLeast& least) {
    static_assert(2 * V <= TY, "the y halo rows are loaded by the first and last V tile rows");
    const int i = i0 + tx, j = j0 + ty;
    const bool inside = i < g.mx && j < g.my;
    const bool ghosted = i < g.mx + V && j < g.my + V;   // own slot of the tiles is read by someone
    const int P = (int)g.P, PS = (int)g.PS;
    const int c0 = (int)g.at(i, j, 0);
    i64 kx, ky, kz;
    fx_theta_factors(b, e, g.nonuniform_x, inside ? xp[i] : 0.0, kx, ky, kz);
    i64 ring[2 * V + 1];
#pragma unroll
    for (int l = 0; l < 2 * V; l++) ring[l] = inside ? fx_from(__ldg(in.w + c0 + (k0 - V + l) * PS), e[3]) : 0;
    double nw = 0., nu = 0., nv = 0., hx = 0., hy = 0.;
    const bool xl = tx < V, xr = tx >= 32 - V, yl = ty < V, yr = ty >= TY - V;
    const auto fetch = [&](int k) {
        const int ck = c0 + k * PS;
        nw = inside ? __ldg(in.w + ck + V * PS) : 0.0;
        if (ghosted) {
            nu = __ldg(in.u + ck);
            nv = __ldg(in.v + ck);
        }
        // the halos: a thread fills at most one of the two x halos and one of the two y halos
        if (xl && j < g.my) hx = __ldg(in.u + ck - V);
        if (xr && i < g.mx && j < g.my) hx = __ldg(in.u + ck + V);
        if (yl && i < g.mx) hy = __ldg(in.v + ck - V * P);
        if (yr && j < g.my && i < g.mx) hy = __ldg(in.v + ck + V * P);
    };
    if (k0 < k1) fetch(k0);
    for (int k = k0; k < k1; k++) {
        const int ck = c0 + k * PS;
        double q[5] = {0, 0, 0, 0, 0};
        if (inside) {
            q[0] = __ldg(in.r + ck); q[1] = __ldg(in.t + ck); q[2] = __ldg(in.p + ck);
            q[3] = __ldg(in.h + ck); q[4] = __ldg(in.m + ck);
        }
        const i64 cu = fx_from(nu, e[1]), cv = fx_from(nv, e[2]);
        ring[2 * V] = fx_from(nw, e[3]);
        const i64 cx = xl || xr ? fx_from(hx, e[1]) : 0, cy = yl || yr ? fx_from(hy, e[2]) : 0;
        if (k + 1 < k1) fetch(k + 1);
        __syncthreads();   // the previous plane's tiles are no longer read
        su[ty][tx + V] = cu;
        sv[ty + V][tx] = cv;
        if (xl) su[ty][tx] = cx;
        if (xr) su[ty][tx + 2 * V] = cx;
        if (yl) sv[ty][tx] = cy;
        if (yr) sv[ty + 2 * V][tx] = cy;
        __syncthreads();
        if (inside) {
            FxSum sx, sy, sz;
#pragma unroll
            for (int l = 1; l <= V; l++) {
                sx.add(su[ty][tx + V + l] - su[ty][tx + V - l], fxw1(V, l));
                sy.add(sv[ty + V + l][tx] - sv[ty + V - l][tx], fxw1(V, l));
                sz.add(ring[V + l] - ring[V - l], fxw1(V, l));
            }
            const i64 th = fx_mul(sx.value(), kx) + fx_mul(sy.value(), ky) + fx_mul(sz.value(), kz);
            in.fx.th[ck] = th;
            if (own) dil_ghost_owner<i64>(g, in.fx.th, ck, i, j, k, th);
            fx_store(in.fx, e, ck, cu, cv, ring[V], q);
            least.add(q[0], q[1]);
        }
#pragma unroll
        for (int l = 0; l < 2 * V; l++) ring[l] = ring[l + 1];
    }
}

// The conversion and theta of one point, every neighbour from global memory (the batched
// stage kernel's form; the same integers)
template <int V>
__device__ __forceinline__ void fx_point(const Geom& g, const FxBase& b, const RhsIn<double>& in, const int (&e)[8],
                                         const double* __restrict__ xp, int i, int j, int k, FxLeast& least) {
    const int c = (int)g.at(i, j, k), P = (int)g.P, PS = (int)g.PS;
    i64 kx, ky, kz;
    fx_theta_factors(b, e, g.nonuniform_x, xp[i], kx, ky, kz);
    FxSum sx, sy, sz;
#pragma unroll
    for (int l = 1; l <= V; l++) {
        sx.add(fx_from(in.u[c + l], e[1]) - fx_from(in.u[c - l], e[1]), fxw1(V, l));
        sy.add(fx_from(in.v[c + l * P], e[2]) - fx_from(in.v[c - l * P], e[2]), fxw1(V, l));
        sz.add(fx_from(in.w[c + l * PS], e[3]) - fx_from(in.w[c - l * PS], e[3]), fxw1(V, l));
    }
    const i64 th = fx_mul(sx.value(), kx) + fx_mul(sy.value(), ky) + fx_mul(sz.value(), kz);
    in.fx.th[c] = th;
    double q[5];
    fx_scan(in, c, q);
    least.add(q[0], q[1]);
    fx_store(in.fx, e, c, fx_from(in.u[c], e[1]), fx_from(in.v[c], e[2]), fx_from(in.w[c], e[3]), q);
}

// The sums of one direction at a point, in two passes over the neighbour pairs (-l, l), each of
// which loads a pair once and feeds every sum that needs it (one pass for all of them needs 150
// registers: 640 bytes spilled and 1.28 against 1.23 ms on the channel; with the four values
// both passes read as one 32-byte load and both loops unrolled 0.88 ms):
//   fx_visc  first derivatives of u, v, w, mu, T, theta and second ones of u, v, w, T (viscous
//            order)
//   fx_conv  first derivative of p and the telescoped split-form fluxes (advective order)
//              sum_l a_l (Q- - Q+)  and  sum_l a_l (Q- phi_{-l} - Q+ phi_l),
//              Q+- = (rho_0 + rho_{+-l}) (g_0 + g_{+-l}),  g the velocity along the direction
// Bounds (F: a field, |F| < 2^62): differences and sums of two fields < 2^63; Q < 2^62; a
// flux term's two sides together < 2^61, their cross products < 2^63 (1 - 2^-21) + 2^33.
struct FxVisc {
    i64 d[6], L[4];   // u, v, w, mu, T, theta; u, v, w, T
};
struct FxConv {
    i64 p, F[5];   // mass flux; u, v, w, H fluxes, doubled
    int ps;        // p is 2^ps times the sum
};

template <int V, bool RO>
__device__ __forceinline__ FxVisc fx_visc(const FxFields& in, int c, int st, const i64 (&ctr)[4]) {
    FxSum D[6], L[4];
#pragma unroll
    for (int q = 0; q < 4; q++) L[q].add(ctr[q], fxw2(V, 0));
#pragma unroll
    for (int l = 1; l <= V; l++) {
        const Fx4 am = fx_load4<RO>(in.v + c - l * st), ap = fx_load4<RO>(in.v + c + l * st);
        const longlong2 tm = ld<RO>(in.t + c - l * st), tp = ld<RO>(in.t + c + l * st);
        D[0].add(ap.x - am.x, fxw1(V, l));
        D[1].add(ap.y - am.y, fxw1(V, l));
        D[2].add(ap.z - am.z, fxw1(V, l));
        D[3].add(tp.y - tm.y, fxw1(V, l));
        D[4].add(tp.x - tm.x, fxw1(V, l));
        D[5].add(ld<RO>(in.th + c + l * st) - ld<RO>(in.th + c - l * st), fxw1(V, l));
        L[0].add(ap.x + am.x, fxw2(V, l));
        L[1].add(ap.y + am.y, fxw2(V, l));
        L[2].add(ap.z + am.z, fxw2(V, l));
        L[3].add(tp.x + tm.x, fxw2(V, l));
    }
    FxVisc o;
#pragma unroll
    for (int q = 0; q < 6; q++) o.d[q] = D[q].value();
#pragma unroll
    for (int q = 0; q < 4; q++) o.L[q] = L[q].value();
    return o;
}

template <int S, int DIR, bool ROLLED, bool RO>
__device__ __forceinline__ FxConv fx_conv(const FxFields& in, int c, int st, i64 r0, i64 g0) {
    FxSum P, F[5];
#pragma unroll(ROLLED ? 1 : S)
    for (int l = 1; l <= S; l++) {
        const Fx4 am = fx_load4<RO>(in.v + c - l * st), ap = fx_load4<RO>(in.v + c + l * st);
        const longlong2 hm = ld<RO>(in.r + c - l * st), hp = ld<RO>(in.r + c + l * st);
        P.add(ap.w - am.w, fxw1(S, l));
        const i64 gm = DIR == 0 ? am.x : DIR == 1 ? am.y : am.z;
        const i64 gp = DIR == 0 ? ap.x : DIR == 1 ? ap.y : ap.z;
        const i64 qm = fx_mul(hm.x + r0, gm + g0), qp = -fx_mul(hp.x + r0, gp + g0);
        F[0].add(qm + qp, fxw1(S, l));
        const int qmh = fx_hi(qm), qml = fx_lo(qm), qph = fx_hi(qp), qpl = fx_lo(qp);
        const i64 phm[4] = {am.x, am.y, am.z, hm.y}, php[4] = {ap.x, ap.y, ap.z, hp.y};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int mh = fx_hi(phm[q]), ml = fx_lo(phm[q]), ph = fx_hi(php[q]), pl = fx_lo(php[q]);
            const i64 m = fx_mad(qmh, ml, fx_mad(qml, mh, fx_mad(qph, pl, fx_mad(qpl, ph, FX_HALF))));
            F[1 + q].add(fx_mad(qmh, mh, fx_mad(qph, ph, (i64)fx_word1(m))), fxw1(S, l));
        }
    }
    FxConv o;
    o.p = P.normal(o.ps);
#pragma unroll
    for (int q = 0; q < 5; q++) o.F[q] = q == 0 ? F[q].value() : F[q].twice();
    return o;
}

// fx_mul with a table factor (low word, balanced high half)
__device__ __forceinline__ i64 fx_mulk(i64 v, i64 k) {
    const int vh = fx_hi(v), vl = fx_lo(v), kh = fx_word1(k), kl = fx_lo(k);
    const i64 m = fx_mad(vh, kl, fx_mad(vl, kh, FX_HALF));
    return fx_mad(vh, kh, (i64)fx_word1(m));
}

// sum of three products / 2^64, the low halves' products (below a quarter each) left out;
// factors below 2^62 and 2^62: the cross sums < 2^62.6 in pairs of products
__device__ __forceinline__ i64 fx_dot3(i64 a0, i64 b0, i64 a1, i64 b1, i64 a2, i64 b2) {
    const int a0h = fx_hi(a0), a1h = fx_hi(a1), a2h = fx_hi(a2), b0h = fx_hi(b0), b1h = fx_hi(b1), b2h = fx_hi(b2);
    const i64 m = fx_mad(a0h, fx_lo(b0), fx_mad(fx_lo(a0), b0h, FX_HALF));
    const i64 n = fx_mad(a1h, fx_lo(b1), fx_mad(fx_lo(a1), b1h, FX_HALF));
    const i64 o = fx_mad(a2h, fx_lo(b2), fx_mad(fx_lo(a2), b2h, FX_HALF));
    return fx_mad(a0h, b0h, fx_mad(a1h, b1h, fx_mad(a2h, b2h, (i64)fx_word1(m) + fx_word1(n) + fx_word1(o))));
}

// table unit q times 2^-s
template <bool RO>
__device__ __forceinline__ double fx_unit(const i64* K, int q, int s) {
    const double k = __longlong_as_double(ld<RO>(K + q));
    return __hiloint2double(__double2hiint(k) - (s << 20), __double2loint(k));
}

// RHS of one interior point at element c (without body force and sponge), in two parts that
// share no intermediate value. Bounds in the units of fx_table: gradients < 2^59.8, theta,
// stress < 2^61.8, grad mu, grad T < 2^60.8, second derivatives < 2^62.3, RHS sums < 2^62.4.
//
// BATCH: the persistent batch kernel's form, the loops over the offsets not unrolled and the
// inputs written by earlier phases of the same launch.
//
// The convective and pressure terms. Neither grad p nor grad theta (fx_viscous) joins an integer
// sum: their largest possible values would set its unit, and where a velocity component is far
// smaller than the others or than the speed of sound, its fluxes and second derivatives would
// lose bits (spanwise velocity 2^-15 of the stream: joined, its equation was off by 7.6e-12 of its
// maximum, FP64 sums 8.9e-14; a stage on the channel 128x160x192 1.15 -> 1.20 ms). dp and the sums meet in FP64
// here, before the viscous part, which holds fewer registers than after it (1.20 against 1.23 ms).
template <int S, bool BATCH>
__device__ __forceinline__ void fx_convective(const Geom& g, const FxBase& b, const FxFields& x, int i, int c,
                                              double (&out)[5]) {
    constexpr bool RO = !BATCH;
    const i64* K = x.k;
    i64 acc[5] = {0, 0, 0, 0, 0};
    double dp[3];
    const bool nux = g.nonuniform_x;
    const i64 xp = nux ? __ldg(b.xpk + i) : 0;
    const Fx4 A = fx_load4<RO>(x.v + c);
    const longlong2 H = ld<RO>(x.r + c);
    const auto conv = [&](const FxConv& o, int d, bool sx) {
        const i64* k = K + d * FXK_DIR;
        const auto f = [&](i64 v, int q) { return fx_mulk(sx ? fx_mulk(v, xp) : v, ld<RO>(k + q)); };
        dp[d] = __dmul_rn((double)(sx ? fx_mulk(o.p, xp) : o.p), fx_unit<RO>(k, FXK_P, o.ps));
#pragma unroll
        for (int q = 0; q < 5; q++) acc[q] += f(o.F[q], FXK_F0 + q);
    };
    conv(fx_conv<S, 0, BATCH, RO>(x, c, 1, H.x, A.x), 0, nux);
    conv(fx_conv<S, 1, BATCH, RO>(x, c, (int)g.P, H.x, A.y), 1, false);
    conv(fx_conv<S, 2, BATCH, RO>(x, c, (int)g.PS, H.x, A.z), 2, false);
    // the cubic fluxes' centre values: phi_0 times half the mass flux
    const i64 phi[4] = {A.x, A.y, A.z, H.y};
#pragma unroll
    for (int q = 0; q < 4; q++) acc[1 + q] += fx_mulk(fx_mul_by4(phi[q], acc[0]), ld<RO>(K + FXK_CTR + q));
#pragma unroll
    for (int q = 0; q < 5; q++) {
        const double v = (double)acc[q], unit = fx_unit<RO>(K, FXK_A + q, 0);
        out[q] = q == 0 || q == 4 ? __dmul_rn(v, unit) : fma(v, unit, -dp[q > 0 ? q - 1 : 0]);
    }
}

// The viscous terms: force in out[0..2], conduction, dissipation and work in out[3]
template <int V, bool BATCH>
__device__ __forceinline__ void fx_viscous(const Geom& g, const FxBase& b, const RhsIn<double>& in, int quirk, int i,
                                           int c, double u0, double v0, double w0, double (&out)[4]) {
    const FxFields& x = in.fx;
    constexpr bool RO = !BATCH;
    const i64* K = x.k;
    const bool nux = g.nonuniform_x;
    const i64 xp = nux ? __ldg(b.xpk + i) : 0;
    const Fx4 A = fx_load4<RO>(x.v + c);
    const longlong2 T = ld<RO>(x.t + c);
    const i64 ctr[4] = {A.x, A.y, A.z, T.x};
    const longlong2 xx = nux ? __ldg(b.xx + i) : make_longlong2(0, 0);
    i64 G[9], dmu[3], dT[3], L[4] = {0, 0, 0, 0};
    // mu/3 grad theta, apart from the second derivatives for the same reason as grad p
    double th[3];
    const auto visc = [&](const FxVisc& o, int d, bool sx) {
        const i64* k = K + d * FXK_DIR;
        const auto f = [&](i64 v, int q) { return fx_mulk(sx ? fx_mulk(v, xp) : v, ld<RO>(k + q)); };
#pragma unroll
        for (int q = 0; q < 3; q++) G[3 * d + q] = f(o.d[q], FXK_U + q);
        dmu[d] = f(o.d[3], FXK_MU);
        dT[d] = f(o.d[4], FXK_T);
#pragma unroll
        for (int q = 0; q < 4; q++)
            L[q] += fx_mulk(sx ? fx_mul2(xx.x, o.L[q], xx.y, o.d[q < 3 ? q : 4]) : o.L[q], ld<RO>(k + FXK_L + q));
        const int s = fx_room(fx_bits(o.d[5]));
        th[d] = __dmul_rn((double)fx_mul(T.y, sx ? fx_mulk(o.d[5] << s, xp) : o.d[5] << s), fx_unit<RO>(k, FXK_TH, s));
    };
    visc(fx_visc<V, RO>(x, c, 1, ctr), 0, nux);
    visc(fx_visc<V, RO>(x, c, (int)g.P, ctr), 1, false);
    visc(fx_visc<V, RO>(x, c, (int)g.PS, ctr), 2, false);
    // grad mu and the stress tensor tau / mu, each scaled to the full range
    const int sm = fx_room(fx_bits(dmu[0]) | fx_bits(dmu[1]) | fx_bits(dmu[2]));
#pragma unroll
    for (int q = 0; q < 3; q++) dmu[q] <<= sm;
    const i64 th3 = fx_mulk(ld<RO>(x.th + c), ld<RO>(K + FXK_TG));   // theta / 3
    i64 t[6] = {2 * (G[0] - th3), 2 * (G[4] - th3), 2 * (G[8] - th3), G[1] + G[3], G[2] + G[6], G[5] + G[7]};
    // y-z dissipation with the quirk: tau_yz dv/dz in the y sum as in the z sum (src/cuda_rhs.cu:175)
    i64 q12 = quirk ? 2 * G[7] : t[5];
    const int st = fx_room(fx_bits(t[0]) | fx_bits(t[1]) | fx_bits(t[2]) | fx_bits(t[3]) | fx_bits(t[4]) |
                           fx_bits(t[5]) | fx_bits(q12));
#pragma unroll
    for (int q = 0; q < 6; q++) t[q] <<= st;
    q12 <<= st;
    // dissipation / mu: tau_ab du_b/dx_a = sum t_aa^2 / 2 (the trace of t is zero) + sum t_ab^2
    const i64 diss = (fx_dot3(t[0], t[0], t[1], t[1], t[2], t[2]) >> 1) + fx_dot3(t[3], t[3], t[4], t[4], t[5], q12);
    const double ud = fx_unit<RO>(K, FXK_UD, sm + st);
    out[0] = fma((double)fx_mul(T.y, L[0]), fx_unit<RO>(K, FXK_UL, 0),
                 fma((double)fx_dot3(t[0], dmu[0], t[3], dmu[1], t[4], dmu[2]), ud, th[0]));
    out[1] = fma((double)fx_mul(T.y, L[1]), fx_unit<RO>(K, FXK_UL + 1, 0),
                 fma((double)fx_dot3(t[3], dmu[0], t[1], dmu[1], t[5], dmu[2]), ud, th[1]));
    out[2] = fma((double)fx_mul(T.y, L[2]), fx_unit<RO>(K, FXK_UL + 2, 0),
                 fma((double)fx_dot3(t[4], dmu[0], t[5], dmu[1], t[2], dmu[2]), ud, th[2]));
    double en = (double)fx_mul(T.y, L[3]) * fx_unit<RO>(K, FXK_UL + 3, 0);
    en = fma((double)fx_dot3(dT[0], dmu[0], dT[1], dmu[1], dT[2], dmu[2]), fx_unit<RO>(K, FXK_UC, sm), en);
    en = fma(in.m[c], (double)diss * fx_unit<RO>(K, FXK_UE, 2 * st), en);
    out[3] = fma(u0, out[0], fma(v0, out[1], fma(w0, out[2], en)));
}

// ---- FP64 sums ----
// theta at element c and its ghost images
template <int V, bool RO>
__device__ __noinline__ void wide_theta(const Geom& g, const CoefT<double>& cf, const RhsIn<double>& in, int i, int j,
                                        int k, bool own) {
    const int c = (int)g.at(i, j, k), P = (int)g.P, PS = (int)g.PS;
    const auto d1 = [&](const double* f, int st, const double* co) {
        double s = co[1] * (ld<RO>(f + c + st) - ld<RO>(f + c - st));
#pragma unroll
        for (int l = 2; l <= V; l++) s = fma(co[l], ld<RO>(f + c + l * st) - ld<RO>(f + c - l * st), s);
        return s;
    };
    double x = d1(in.u, 1, cf.c1V[0]);
    if (g.nonuniform_x) x *= cf.xp[i];
    const double th = x + d1(in.v, P, cf.c1V[1]) + d1(in.w, PS, cf.c1V[2]);
    double* o = (double*)in.fx.th;
    o[c] = th;
    if (own) dil_ghost_owner<double>(g, o, c, i, j, k, th);
}

// RHS of the point at element c (without body force and sponge), with the sums of fx_convective
// and fx_viscous in FP64 from the FP64 fields and theta
template <int S, int V, bool RO>
__device__ __forceinline__ void rhs_wide(const Geom& g, const CoefT<double>& cf, const RhsIn<double>& in, int quirk,
                                         int i, int c, double (&acc)[5]) {
    const double* th = (const double*)in.fx.th;
    const auto at = [&](const double* f, int o) { return ld<RO>(f + c + o); };
    const bool nux = g.nonuniform_x;
    const double xp = nux ? cf.xp[i] : 1.0;
    const double u0 = at(in.u, 0), v0 = at(in.v, 0), w0 = at(in.w, 0), r0 = at(in.r, 0), h0 = at(in.h, 0),
                 m0 = at(in.m, 0), th23 = (2. / 3.) * at(th, 0);
    const auto d1 = [&](const double* f, int st, const double* co) {
        double s = co[1] * (at(f, st) - at(f, -st));
#pragma unroll
        for (int l = 2; l <= V; l++) s = fma(co[l], at(f, l * st) - at(f, -l * st), s);
        return s;
    };
    double G[9];   // G[3 a + b] = d u_b / d x_a
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int st = d == 0 ? 1 : (int)(d == 1 ? g.P : g.PS);
        const double x = d == 0 ? xp : 1.0;
        G[3 * d] = d1(in.u, st, cf.c1V[d]) * x;
        G[3 * d + 1] = d1(in.v, st, cf.c1V[d]) * x;
        G[3 * d + 2] = d1(in.w, st, cf.c1V[d]) * x;
    }
    const double t[6] = {fma(2.0, G[0], -th23), fma(2.0, G[4], -th23), fma(2.0, G[8], -th23),
                         G[1] + G[3], G[2] + G[6], G[5] + G[7]};
    // y-z dissipation with the quirk: tau_yz dv/dz in the y sum as in the z sum (src/cuda_rhs.cu:175)
    const double q12 = quirk ? G[7] + G[7] : t[5];
    const double diss = fma(t[0], G[0], fma(t[1], G[4], fma(t[2], G[8], fma(t[3], t[3], fma(t[4], t[4], t[5] * q12)))));
#pragma unroll
    for (int q = 0; q < 5; q++) acc[q] = 0.0;
    double W[3] = {0, 0, 0}, L[4] = {0, 0, 0, 0}, cond = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int st = d == 0 ? 1 : (int)(d == 1 ? g.P : g.PS);
        const bool sx = d == 0 && nux;
        const double x = sx ? xp : 1.0;
        const double* F[4] = {in.u, in.v, in.w, in.t};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (sx) {
#pragma unroll
                for (int l = -V; l <= V; l++) L[q] = fma(__ldg(cf.cvsx + (l + V) * g.mx + i), at(F[q], l), L[q]);
            } else {
                L[q] = fma(cf.c2V[d][0], at(F[q], 0), L[q]);
#pragma unroll
                for (int l = 1; l <= V; l++) L[q] = fma(cf.c2V[d][l], at(F[q], l * st) + at(F[q], -l * st), L[q]);
            }
        }
        const double dmu = d1(in.m, st, cf.c1V[d]) * x;
        W[0] = fma(d == 0 ? t[0] : d == 1 ? t[3] : t[4], dmu, W[0]);
        W[1] = fma(d == 0 ? t[3] : d == 1 ? t[1] : t[5], dmu, W[1]);
        W[2] = fma(d == 0 ? t[4] : d == 1 ? t[5] : t[2], dmu, W[2]);
        cond = fma(d1(in.t, st, cf.c1V[d]) * x, dmu, cond);
        W[d] = fma(m0 * (1.0 / 3.0), d1(th, st, cf.c1V[d]) * x, W[d]);
        // fluxes (fx_conv's) and the pressure gradient; fc = c1S / 4, the mass flux's weight twice that
        const double* gf = d == 0 ? in.u : d == 1 ? in.v : in.w;
        const double g0 = d == 0 ? u0 : d == 1 ? v0 : w0;
        double f[5] = {0, 0, 0, 0, 0}, dp = 0.0;
#pragma unroll
        for (int l = 1; l <= S; l++) {
            const double am = cf.fc[d][l] * (at(in.r, -l * st) + r0) * (at(gf, -l * st) + g0);
            const double ap = cf.fc[d][l] * (r0 + at(in.r, l * st)) * (g0 + at(gf, l * st));
            f[0] += am - ap;
            f[1] = fma(am, at(in.u, -l * st), fma(-ap, at(in.u, l * st), f[1]));
            f[2] = fma(am, at(in.v, -l * st), fma(-ap, at(in.v, l * st), f[2]));
            f[3] = fma(am, at(in.w, -l * st), fma(-ap, at(in.w, l * st), f[3]));
            f[4] = fma(am, at(in.h, -l * st), fma(-ap, at(in.h, l * st), f[4]));
            dp = fma(cf.c1S[d][l], at(in.p, l * st) - at(in.p, -l * st), dp);
        }
        acc[0] = fma(2.0 * x, f[0], acc[0]);
#pragma unroll
        for (int q = 1; q < 5; q++) acc[q] = fma(x, f[q], acc[q]);
        acc[1 + d] = fma(-x, dp, acc[1 + d]);
    }
    const double half = 0.5 * acc[0];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        W[q] = fma(m0, L[q], W[q]);
        acc[1 + q] = fma(q == 0 ? u0 : q == 1 ? v0 : w0, half, acc[1 + q]) + W[q];
    }
    cond = fma(m0, L[3], cond);
    acc[4] = fma(h0, half, acc[4]) + fma(m0, diss, cf.lam_mu * cond) + fma(u0, W[0], fma(v0, W[1], w0 * W[2]));
}

}  // namespace cns
