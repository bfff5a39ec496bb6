// kernels_rhs.cuh -- the RHS + Runge-Kutta stage kernel (one thread per grid point).
//
// Per point it forms the x, y and z contributions of deviceRHSX/Y/Z
// (src/cuda_rhs.cu:9-396), the body force, the sponge (src/sponge.cu:31-41) and then
// the stage update of the selected time scheme (sumLowStorageRK3 + deviceMul/deviceDiv,
// src/cuda_main.cu:109-186,244-247; eulerSum*/rk3final*, src/cuda_main.cu:188-216),
// writing the new state to the other state buffer. All neighbour reads hit the ghosted
// layout, so there is no boundary branching.
//
// The split-form convective derivative is evaluated in its telescoped form. The
// reference accumulates the two interface fluxes F_{i+1/2}, F_{i-1/2} over every
// (l, m) pair of the Kennedy-Gruber sum (src/cuda_derivs.h:30-155) and differences
// them; all pairs except (i-l, i) and (i, i+l) cancel exactly, so
//   d(f g h)/dx |_i = c/dx * sum_l a_l [ P(i-l, i) - P(i, i+l) ],
//   P(a, b) = (f_a + f_b)(g_a + g_b)(h_a + h_b),  a_l = -coeffF[S-l],  c = 1/2 (two
//   factors) or 1/4 (three factors),
// which is the same value with 2 instead of l(l+1) pair products per l. The product
// (rho_a+rho_b)(g_a+g_b) is shared by the mass flux and the four cubic fluxes.
//
// FP64 and pair mode: the sums over the neighbours in 64-bit fixed point, or in FP64 where the
// fields' ranges ask for it (kernels_fx.cuh), the stage update and the recovery in FP64. FP32-RHS mode: rhs_point_packed on FP32 records.
#pragma once
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "cns_common.cuh"
#include "cns_internal.h"
#include "kernels_fx.cuh"
#include "kernels_point.cuh"

namespace cns {

// Body force, sponge, stage update and the new state's recovery of the point at element
// c, given its RHS accumulators acc (convective, pressure and viscous terms) and centre
// values u0, v0, w0, r0 in the arithmetic type R
template <typename R>
__device__ __forceinline__ void stage_tail(const Geom& g, const Update<R>& up, double* __restrict__ scal, int i, int k,
                                           int c, R (&acc)[5], R u0, R v0, R w0, R r0) {
    // ---- body force and sponge (RHS terms, arithmetic type R) ----
    const R dpdz = to_r<R>(scal[SC_DPDZ]);
    acc[3] += dpdz;
    acc[4] = fma(dpdz, w0, acc[4]);
    const double rr = up.qin.r[c], uu = up.qin.u[c], vv = up.qin.v[c], ww = up.qin.w[c], ee = up.qin.e[c];
    if (up.spx) {
        const R sg = to_r<R>(up.spx[i] + up.spz[k]);
        const long long i2 = (long long)i + (long long)k * g.mx;
        if constexpr (sizeof(R) == 8) {
            acc[0] += sg * (up.rref[i2] - rr);
            acc[1] += sg * (up.uref[i2] - rr * uu);
            acc[2] += sg * (up.vref[i2] - rr * vv);
            acc[3] += sg * (up.wref[i2] - rr * ww);
            acc[4] += sg * (up.eref[i2] - ee);
        } else {
            acc[0] += sg * (to_r<R>(up.rref[i2]) - r0);
            acc[1] += sg * (to_r<R>(up.uref[i2]) - r0 * u0);
            acc[2] += sg * (to_r<R>(up.vref[i2]) - r0 * v0);
            acc[3] += sg * (to_r<R>(up.wref[i2]) - r0 * w0);
            acc[4] += sg * (to_r<R>(up.eref[i2]) - to_r<R>(ee));
        }
    }
    if (up.kind == ST_RHS_ONLY) {
#pragma unroll
        for (int q = 0; q < 5; q++) up.rb[q][c] = acc[q];
        return;
    }
    // ---- stage update: the RHS combination in R, the accumulation into the state in FP64 ----
    // The register arrays are read in full before any of them is written: the compiler
    // cannot prove that rb[q] and rb[q+1] (or k2) do not overlap, so interleaved
    // load/store pairs would serialise five memory round trips at the end of every thread.
    const double dt = scal[SC_DT];
    double qn[5];
    if (up.kind == ST_LS) {
        const double q0[5] = {rr, uu * rr, vv * rr, ww * rr, ee};
        const R a = up.ca, b = up.cb;
        R prev[5] = {0, 0, 0, 0, 0};
        if (up.use_prev) {
#pragma unroll
            for (int q = 0; q < 5; q++) prev[q] = up.rb[q][c];
        }
        if constexpr (sizeof(R) == 8) {
            // q0 + dt (a prev + b acc) with dt a, dt b formed once: two operations per field
            const double dta = dt * up.a, dtb = dt * up.b;
#pragma unroll
            for (int q = 0; q < 5; q++) {
                qn[q] = fma(dtb, to_d<R>(acc[q]), up.use_prev ? fma(dta, to_d<R>(prev[q]), q0[q]) : q0[q]);
                up.rb[q][c] = acc[q];
            }
        } else {
#pragma unroll
            for (int q = 0; q < 5; q++) {
                const R x = up.use_prev ? fma(a, prev[q], b * acc[q]) : b * acc[q];
                qn[q] = fma(dt, to_d<R>(x), q0[q]);
                up.rb[q][c] = acc[q];
            }
        }
    } else if (up.kind == ST_C1 || up.kind == ST_R4_1) {
        const double q0[5] = {rr, rr * uu, rr * vv, rr * ww, ee};
#pragma unroll
        for (int q = 0; q < 5; q++) {
            up.q0[q][c] = q0[q];
            const double Rd = to_d<R>(acc[q]);
            if (up.kind == ST_C1) { qn[q] = q0[q] + Rd * dt / 2.0; up.rb[q][c] = acc[q]; }
            else { qn[q] = q0[q] + 0.5 * dt * Rd; up.k2[q][c] = acc[q]; }
        }
    } else {
        double q0[5];
        R k1[5] = {0, 0, 0, 0, 0}, kk[5] = {0, 0, 0, 0, 0};
        const bool use_k1 = up.kind == ST_C2 || up.kind == ST_C3, use_k2 = up.kind != ST_C2;
#pragma unroll
        for (int q = 0; q < 5; q++) {
            q0[q] = up.q0[q][c];
            if (use_k1) k1[q] = up.rb[q][c];
            if (use_k2) kk[q] = up.k2[q][c];
        }
#pragma unroll
        for (int q = 0; q < 5; q++) {
            const double Rd = to_d<R>(acc[q]);
            switch (up.kind) {
            case ST_C2: qn[q] = q0[q] + (2 * Rd - to_d<R>(k1[q])) * dt; up.k2[q][c] = acc[q]; break;
            case ST_C3: qn[q] = q0[q] + dt * (to_d<R>(k1[q]) + 4 * to_d<R>(kk[q]) + Rd) / 6.; break;
            case ST_R4_2: up.k2[q][c] = to_r<R>(to_d<R>(kk[q]) + 2.0 * Rd); qn[q] = q0[q] + 0.5 * dt * Rd; break;
            case ST_R4_3: up.k2[q][c] = to_r<R>(to_d<R>(kk[q]) + 2.0 * Rd); qn[q] = q0[q] + dt * Rd; break;
            default: qn[q] = q0[q] + dt / 6.0 * (to_d<R>(kk[q]) + Rd); break;
            }
        }
    }
    const double inv = rcp_nr(qn[0]);
    const double un = qn[1] * inv, vn = qn[2] * inv, wn = qn[3] * inv;
    up.qout.r[c] = qn[0];
    up.qout.u[c] = un;
    up.qout.v[c] = vn;
    up.qout.w[c] = wn;
    up.qout.e[c] = qn[4];
    // the next stage's state recovery from the values in registers (bit for bit the state
    // kernel's result on the stored state)
    if (up.fuse) state_store<R>(up.ph, up.dnext, scal, c, qn[0], inv, un, vn, wn, qn[4]);
}

// ---------------------------------------------------------------------------------
// FP32-RHS point body on the packed stencil records qa = (rho, u, v, w), qb = (T, p, H, mu)
// and theta. One pass per direction walks the offsets l = 1..S once: at each l it loads
// the two records on either side (four 16-byte loads) and theta (for l <= V) and feeds
// every sum that needs them -- the first derivatives of u, v, w, mu, T, theta at the
// viscous order and of p at the advective order, the second derivatives of u, v, w, T, and
// the telescoped split-form fluxes -- so no stencil is held in registers. Each sum is
// accumulated from the centre term with l ascending; the non-uniform x second derivative adds
// the pair (l, -l) per l.
// ---------------------------------------------------------------------------------
//
// CW (compile-time weights): the sums use the central-difference weights as immediates and
// are scaled by the direction's inverse spacing (or its square) afterwards; the flux sums
// carry neither 1/2, 1/4 nor 1/dx, which the final combination applies. The batched stage
// kernel uses this form: its members' coefficients would otherwise come through shared
// memory and occupy registers. There the inputs are also written by earlier phases of the same
// launch, so this form loads them by ordinary loads (ld, fx.cuh). The standalone kernel reads the premultiplied tables from
// its launch parameters (constant bank operands).
template <int S, int V, int DIR, bool CW>
__device__ __forceinline__ void rhs_dir_packed(const Geom& g, const CoefT<float>& cf, const RhsIn<float>& in, int c,
                                               int st, int i, float (&Gr)[9], float m0, float m3, float u0, float v0,
                                               float w0, float r0, float h0, float T0, float (&acc)[5],
                                               float (&W)[3], float& cond, float& dmu_dir) {
    static_assert(V <= S, "the viscous half-width never exceeds the advective one");
    const bool nux = (DIR == 0) && g.nonuniform_x;
    const float xpi = nux ? cf.xp[i] : 1.0f;
    const float* c1V = cf.c1V[DIR];
    const float* c1S = cf.c1S[DIR];
    const float* c2V = cf.c2V[DIR];
    const float* fq = cf.fq[DIR];
    const float* fcb = cf.fc[DIR];
    const auto w1V = [&](int l) { if constexpr (CW) return fd1(V, l); else return c1V[l]; };
    const auto w1S = [&](int l) { if constexpr (CW) return fd1(S, l); else return c1S[l]; };
    const auto w2V = [&](int l) { if constexpr (CW) return fd2(V, l); else return c2V[l]; };
    const auto wq = [&](int l) { if constexpr (CW) return fd1(S, l); else return fq[l]; };
    const auto wc = [&](int l) { if constexpr (CW) return fd1(S, l); else return fcb[l]; };
    const float un = DIR == 0 ? u0 : (DIR == 1 ? v0 : w0);

    float gu = 0.f, gv = 0.f, gw = 0.f, dmu = 0.f, dT = 0.f, dth = 0.f, dp = 0.f;
    float d2uu, d2vv, d2ww, d2tt;
    if (nux) {
        const float cw = __ldg(cf.cvsx + V * g.mx + i);
        d2uu = cw * u0; d2vv = cw * v0; d2ww = cw * w0; d2tt = cw * T0;
    } else {
        d2uu = w2V(0) * u0; d2vv = w2V(0) * v0; d2ww = w2V(0) * w0; d2tt = w2V(0) * T0;
    }
    float sq = 0.f, fu = (nux || CW) ? 0.f : acc[1], fv = (nux || CW) ? 0.f : acc[2],
          fw = (nux || CW) ? 0.f : acc[3], fe = (nux || CW) ? 0.f : acc[4];
#pragma unroll
    for (int l = 1; l <= S; l++) {
        const float4 Ap = ld<!CW>(in.qa + c + l * st), Am = ld<!CW>(in.qa + c - l * st);
        const float4 Bp = ld<!CW>(in.qb + c + l * st), Bm = ld<!CW>(in.qb + c - l * st);
        if (l <= V) {
            const float thp = ld<!CW>(in.dil + c + l * st), thm = ld<!CW>(in.dil + c - l * st);
            if (l == 1) {
                gu = w1V(1) * (Ap.y - Am.y); gv = w1V(1) * (Ap.z - Am.z); gw = w1V(1) * (Ap.w - Am.w);
                dmu = w1V(1) * (Bp.w - Bm.w); dT = w1V(1) * (Bp.x - Bm.x); dth = w1V(1) * (thp - thm);
            } else {
                gu = fma(w1V(l), Ap.y - Am.y, gu); gv = fma(w1V(l), Ap.z - Am.z, gv);
                gw = fma(w1V(l), Ap.w - Am.w, gw);
                dmu = fma(w1V(l), Bp.w - Bm.w, dmu); dT = fma(w1V(l), Bp.x - Bm.x, dT);
                dth = fma(w1V(l), thp - thm, dth);
            }
            if (nux) {
                const float cp = __ldg(cf.cvsx + (V + l) * g.mx + i), cm = __ldg(cf.cvsx + (V - l) * g.mx + i);
                d2uu = fma(cp, Ap.y, fma(cm, Am.y, d2uu));
                d2vv = fma(cp, Ap.z, fma(cm, Am.z, d2vv));
                d2ww = fma(cp, Ap.w, fma(cm, Am.w, d2ww));
                d2tt = fma(cp, Bp.x, fma(cm, Bm.x, d2tt));
            } else {
                d2uu = fma(w2V(l), Ap.y + Am.y, d2uu);
                d2vv = fma(w2V(l), Ap.z + Am.z, d2vv);
                d2ww = fma(w2V(l), Ap.w + Am.w, d2ww);
                d2tt = fma(w2V(l), Bp.x + Bm.x, d2tt);
            }
        }
        dp = l == 1 ? w1S(1) * (Bp.y - Bm.y) : fma(w1S(l), Bp.y - Bm.y, dp);
        // telescoped split-form fluxes, a_l Q+- shared by the cubic ones
        const float gm = DIR == 0 ? Am.y : (DIR == 1 ? Am.z : Am.w);
        const float gp = DIR == 0 ? Ap.y : (DIR == 1 ? Ap.z : Ap.w);
        const float Qm = (Am.x + r0) * (gm + un);
        const float Qp = (r0 + Ap.x) * (un + gp);
        sq = fma(wq(l), Qm - Qp, sq);
        const float am = wc(l) * Qm, ap = wc(l) * Qp;
        fu = fma(am, Am.y, fma(-ap, Ap.y, fu));
        fv = fma(am, Am.z, fma(-ap, Ap.z, fv));
        fw = fma(am, Am.w, fma(-ap, Ap.w, fw));
        fe = fma(am, Bm.z, fma(-ap, Bp.z, fe));
    }
    // first derivatives: x' on a non-uniform x; with CW also the inverse spacing
    const float s1 = CW ? cf.inv[DIR] * xpi : xpi;
    if (nux || CW) { gu *= s1; gv *= s1; gw *= s1; }
    Gr[3 * DIR + 0] = gu; Gr[3 * DIR + 1] = gv; Gr[3 * DIR + 2] = gw;
    if (CW && !nux) {
        const float s2 = cf.inv2[DIR];
        d2uu *= s2; d2vv *= s2; d2ww *= s2; d2tt *= s2;
    }
    dmu *= s1;
    dmu_dir = dmu;
    W[0] = fma(d2uu, m0, W[0]);
    W[1] = fma(d2vv, m0, W[1]);
    W[2] = fma(d2ww, m0, W[2]);
    // heat conduction (lambda / mu)(mu d2T + dmu dT), the ratio applied once per point
    dT *= s1;
    cond = fma(d2tt, m0, cond);
    cond = fma(dT, dmu, cond);
    dth *= s1;
    dp *= s1;
    W[DIR] = fma(m3, dth, W[DIR]);
    if constexpr (CW) {
        // fluxes: mass c/dx * sq with c = 1/2, the cubic ones c/dx (f + phi_0 sq) with c = 1/4
        const float q2 = 0.5f * s1, q4 = 0.25f * s1;
        acc[0] = fma(q2, sq, acc[0]);
        acc[1] = fma(q4, fma(u0, sq, fu), acc[1]);
        acc[2] = fma(q4, fma(v0, sq, fv), acc[2]);
        acc[3] = fma(q4, fma(w0, sq, fw), acc[3]);
        acc[4] = fma(q4, fma(h0, sq, fe), acc[4]);
    } else {
        const float half = 0.5f * sq;
        fu = fma(u0, half, fu);
        fv = fma(v0, half, fv);
        fw = fma(w0, half, fw);
        fe = fma(h0, half, fe);
        const float fr = nux ? sq : acc[0] + sq;
        if (nux) {
            acc[0] = fma(xpi, fr, acc[0]);
            acc[1] = fma(xpi, fu, acc[1]);
            acc[2] = fma(xpi, fv, acc[2]);
            acc[3] = fma(xpi, fw, acc[3]);
            acc[4] = fma(xpi, fe, acc[4]);
        } else {
            acc[0] = fr; acc[1] = fu; acc[2] = fv; acc[3] = fw; acc[4] = fe;
        }
    }
    acc[1 + DIR] -= dp;
}

template <int S, int V, bool CW>
__device__ __forceinline__ void rhs_point_packed(const Geom& g, const CoefT<float>& cf, const RhsIn<float>& in,
                                                 const Update<float>& up, double* __restrict__ scal, int quirk, int i,
                                                 int j, int k) {
    const int c = (int)g.at(i, j, k);
    const float4 A0 = ld<!CW>(in.qa + c), B0 = ld<!CW>(in.qb + c);
    const float th0 = ld<!CW>(in.dil + c);
    const float r0 = A0.x, u0 = A0.y, v0 = A0.z, w0 = A0.w;
    const float T0 = B0.x, h0 = B0.z, m0 = B0.w;
    const float m3 = m0 * (float)(1.0 / 3.0);
    float Gr[9];
    float acc[5] = {0, 0, 0, 0, 0};
    float W[3] = {0, 0, 0};
    float diss = 0, cond = 0;
    float dmu[3];
    rhs_dir_packed<S, V, 0, CW>(g, cf, in, c, 1, i, Gr, m0, m3, u0, v0, w0, r0, h0, T0, acc, W, cond, dmu[0]);
    rhs_dir_packed<S, V, 1, CW>(g, cf, in, c, (int)g.P, i, Gr, m0, m3, u0, v0, w0, r0, h0, T0, acc, W, cond, dmu[1]);
    rhs_dir_packed<S, V, 2, CW>(g, cf, in, c, (int)g.PS, i, Gr, m0, m3, u0, v0, w0, r0, h0, T0, acc, W, cond,
                                dmu[2]);
    // stress rows, dissipation and grad(mu) . s of every direction, now that all nine
    // gradients are known (y: tau_yz dv/dz with the quirk, src/cuda_rhs.cu:175)
#pragma unroll
    for (int d = 0; d < 3; d++) {
        float tau[3];
#pragma unroll
        for (int q = 0; q < 3; q++)
            tau[q] = (q == d) ? 2.0f * Gr[3 * d + q] - (float)(2. / 3.) * th0 : Gr[3 * d + q] + Gr[3 * q + d];
        const float dw = (d == 1 && quirk) ? Gr[7] : Gr[3 * d + 2];
        diss = fma(tau[0], Gr[3 * d + 0], diss);
        diss = fma(tau[1], Gr[3 * d + 1], diss);
        diss = fma(tau[2], dw, diss);
        W[0] = fma(tau[0], dmu[d], W[0]);
        W[1] = fma(tau[1], dmu[d], W[1]);
        W[2] = fma(tau[2], dmu[d], W[2]);
    }
    acc[1] += W[0];
    acc[2] += W[1];
    acc[3] += W[2];
    acc[4] += fma(m0, diss, cf.lam_mu * cond) + fma(u0, W[0], fma(v0, W[1], w0 * W[2]));
    stage_tail<float>(g, up, scal, i, k, c, acc, u0, v0, w0, r0);
}

// The FP64 mode's point of a stage with FP64 sums (a call of its own: the other path keeps its
// registers)
template <int S, int V, bool RO>
__device__ __noinline__ void wide_point(const Geom& g, const CoefT<double>& cf, const RhsIn<double>& in,
                                        const Update<double>& up, double* scal, int quirk, int i, int j, int k) {
    const int c = (int)g.at(i, j, k);
    double acc[5];
    rhs_wide<S, V, RO>(g, cf, in, quirk, i, c, acc);
    stage_tail<double>(g, up, scal, i, k, c, acc, up.qin.u[c], up.qin.v[c], up.qin.w[c], up.qin.r[c]);
}

// RHS + stage update of one interior point (i, j, k), every neighbour from global memory
// (CW: the FP32 body with compile-time weights, see rhs_dir_packed)
template <typename R, int S, int V, bool CW = false>
__device__ __forceinline__ void rhs_point(const Geom& g, const CoefT<R>& cf, const RhsIn<R>& in, const Update<R>& up,
                                          double* __restrict__ scal, int quirk, int i, int j, int k) {
    if constexpr (sizeof(R) == 4) {
        rhs_point_packed<S, V, CW>(g, cf, in, up, scal, quirk, i, j, k);
    } else {
        if (ld<!CW>(in.fx.k + FXK_WIDE) != 0) {
            wide_point<S, V, !CW>(g, cf, in, up, scal, quirk, i, j, k);
            return;
        }
        const int c = (int)g.at(i, j, k);
        const double u0 = up.qin.u[c], v0 = up.qin.v[c], w0 = up.qin.w[c];
        double acc[5];
        double vis[4];
        fx_convective<S, CW>(g, cf.fx, in.fx, i, c, acc);
        fx_viscous<V, CW>(g, cf.fx, in, quirk, i, c, u0, v0, w0, vis);
#pragma unroll
        for (int q = 0; q < 4; q++) acc[1 + q] = __dadd_rn(acc[1 + q], vis[q]);
        stage_tail<double>(g, up, scal, i, k, c, acc, u0, v0, w0, up.qin.r[c]);
    }
}

// One launch covers the rows [row0, row0 + gridDim.y * rows per block) of every plane; blocks are
// dispatched x fastest, then rows, then planes. On large planes the rows are split into groups
// launched one after another, so the planes a z stencil spans stay in L2 while a group's blocks
// sweep them (one launch over whole planes would cycle ~2S planes of the inputs through L2
// between their uses).
//
// FP32: 7 blocks of 128 per SM (72 registers) measured fastest (6: 80 registers, +13 %
// time; 5: 96 registers, and stages that read the RK register ran 3.5x slower). FP64: 4 blocks
// (128 registers), bound by latency: issue 37 %, FP64 pipe 50 %, ~3,890 instructions per point,
// 0.995 ms on the channel 128x160x192 (when that was 0.93 ms, before grad p and grad theta left the
// integer sums, 3 blocks of 168 registers took 1.11, 5 of 96, spilling, 0.98).
template <typename R, int S, int V>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 7 : 4) k_rhs(const __grid_constant__ Geom g,
                                                                     const __grid_constant__ CoefT<R> cf,
                                                                     const __grid_constant__ RhsIn<R> in,
                                                                     const __grid_constant__ Update<R> up,
                                                                     double* __restrict__ scal, int quirk, int row0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = row0 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
    if (i >= g.mx || j >= g.my) return;
    rhs_point<R, S, V>(g, cf, in, up, scal, quirk, i, j, (int)blockIdx.z);
}

// FP64 on boxes with at most one block of k_rhs per SM, where a thread's dependent chain is the
// kernel's time: a point takes two threads. The first half of a block's warps form the
// convective part of its 64 points (32 x 2, or 16 x 4 on a narrow box) and, with the viscous part that the other warps hand over
// in shared memory, the stage update. 14^3 .. 28^3 boxes 14.3 .. 16.4 us against 16.4 .. 18.4; from
// 32^3 (18.8 us against 18.4) on one thread per point is the faster, on the channel 128x160x192
// 0.93 ms against 1.12 (measured before grad p and grad theta left the integer sums; a 16x20x24
// box's kernel still takes 14.3 us).
constexpr int SPLIT_POINTS = 64;
template <int S, int V>
__global__ void __launch_bounds__(2 * SPLIT_POINTS, 4) k_rhs_split(const __grid_constant__ Geom g,
                                                                  const __grid_constant__ CoefT<double> cf,
                                                                  const __grid_constant__ RhsIn<double> in,
                                                                  const __grid_constant__ Update<double> up,
                                                                  double* __restrict__ scal,
                                                                  int quirk) {
    __shared__ double sv[4][SPLIT_POINTS];
    const int bh = (int)blockDim.y / 2, row = (int)threadIdx.y % bh, s = row * (int)blockDim.x + (int)threadIdx.x;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = (int)blockIdx.y * bh + row, k = (int)blockIdx.z;
    const bool inside = i < g.mx && j < g.my, first = (int)threadIdx.y < bh;
    const int c = (int)g.at(i, j, k);
    if (ld<true>(in.fx.k + FXK_WIDE) != 0) {
        if (inside && first) wide_point<S, V, true>(g, cf, in, up, scal, quirk, i, j, k);
        return;
    }
    double acc[5];
    if (inside) {
        if (first) {
            fx_convective<S, false>(g, cf.fx, in.fx, i, c, acc);
        } else {
            double vis[4];
            fx_viscous<V, false>(g, cf.fx, in, quirk, i, c, up.qin.u[c], up.qin.v[c], up.qin.w[c], vis);
#pragma unroll
            for (int q = 0; q < 4; q++) sv[q][s] = vis[q];
        }
    }
    __syncthreads();
    if (!inside || !first) return;
#pragma unroll
    for (int q = 0; q < 4; q++) acc[1 + q] = __dadd_rn(acc[1 + q], sv[q][s]);
    stage_tail<double>(g, up, scal, i, k, c, acc, up.qin.u[c], up.qin.v[c], up.qin.w[c], up.qin.r[c]);
}

// Bands per launch: all of them while 3 S planes of a band group at 72 B per point (the
// stencil inputs of the FP64 kernel; twice the FP32 kernel's, whose other traffic streams
// through L2 alongside) fit in half of L2, else the largest group that does (at least 8
// bands). Measured on a 512^3 channel, FP32 RHS step: one launch 45.1 ms, groups of 75
// bands 38.6, 37 bands 36.9, 18 bands 36.9, 9 bands 37.3 ms; on 256^3 one launch (this
// rule) 4.64 ms, groups of 37 bands 4.69, 18 bands 4.74 ms. FP64, a stage on 512 x 512 x 96: one
// launch 6.75 ms, this rule 5.91.
inline int rhs_band_group(const Geom& g) {
    const int nby = (g.my + 3) / 4;
    const size_t budget = (size_t)64 << 20, per_band = (size_t)3 * g.G * g.mx * 4 * 72;
    const size_t fit = budget / per_band;
    if (fit >= (size_t)nby) return nby;
    return fit < 8 ? 8 : (int)fit;
}

// Block of up to `threads` threads over an x-y plane: bw columns, a tile width that divides mx
// into equal parts (12 <= bw <= 64 unless mx is smaller), and bh rows, with the fewest warps for
// the plane and, among equals, bw nearest 32; 32 columns unless that saves 5 % of the warps
// (rows of 32 coalesce best: 150 x 91 is 2 to 6 % slower in 25 columns at 1 % fewer warps). Fixed
// 32 x 4 tiles left 24 % of the lanes idle on a 75 x 53 plane, 25 % at mx = 72 or 48, half at 16:
// FP64 RHS of 72x20x320 158 -> 135 us, 100^3 301 -> 259, 40^3 37 -> 26; FP32 48^3 18.4 -> 14.3.
struct PlaneTile {
    int bw, bh;
};
inline PlaneTile plane_tile(int mx, int my, int threads) {
    PlaneTile best{32, threads / 32};
    const long long wide = (long long)((mx + 31) / 32) * ((my + best.bh - 1) / best.bh) * best.bh;   // in 32 columns
    long long cost = wide * 19 / 20;
    for (int n = (mx + 63) / 64; n <= (mx + 11) / 12; n++) {
        const int bw = (mx + n - 1) / n, bh = std::min(threads / bw, my);
        const long long c = (long long)((mx + bw - 1) / bw) * ((my + bh - 1) / bh) * ((bw * bh + 31) / 32);
        if (c < cost || (c == cost && std::abs(bw - 32) < std::abs(best.bw - 32))) {
            cost = c;
            best = PlaneTile{bw, bh};
        }
    }
    return best;
}

// f(S, V) with the orders as integral constants; false: no such instantiation
template <class F>
bool rhs_dispatch(int S, int V, F f) {
#define CNS_RHS_CASE(SS, VV)                                                               \
    if (S == SS && V == VV) {                                                              \
        f(std::integral_constant<int, SS>(), std::integral_constant<int, VV>());           \
        return true;                                                                       \
    }
    CNS_RHS_CASE(1, 1)
    CNS_RHS_CASE(2, 1) CNS_RHS_CASE(2, 2)
    CNS_RHS_CASE(3, 1) CNS_RHS_CASE(3, 2) CNS_RHS_CASE(3, 3)
    CNS_RHS_CASE(4, 1) CNS_RHS_CASE(4, 2) CNS_RHS_CASE(4, 3) CNS_RHS_CASE(4, 4)
#undef CNS_RHS_CASE
    return false;
}

template <typename R>
int launch_rhs_t(int S, int V, const Geom& g, const CoefT<R>& cf, const RhsIn<R>& in, const Update<R>& up,
                 double* scal, int quirk, cudaStream_t s) {
    const PlaneTile t = plane_tile(g.mx, g.my, 128);
    const int rows = (4 * rhs_band_group(g) + t.bh - 1) / t.bh * t.bh;   // per launch
    int n = 0;
    for (int j0 = 0; j0 < g.my; j0 += rows, n++) {
        const int r = g.my - j0 < rows ? g.my - j0 : rows;
        const dim3 grid((g.mx + t.bw - 1) / t.bw, (r + t.bh - 1) / t.bh, g.mz), block(t.bw, t.bh, 1);
        if (!rhs_dispatch(S, V, [&](auto s_, auto v_) {
                k_rhs<R, decltype(s_)::value, decltype(v_)::value><<<grid, block, 0, s>>>(g, cf, in, up, scal, quirk, j0);
            }))
            break;
    }
    return n;
}

}  // namespace cns
