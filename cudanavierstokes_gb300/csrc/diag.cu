// diag.cu -- volume-averaged viscous dissipation and enstrophy of the current state:
//   eps = < tau_ij du_i/dx_j >,  tau_ij = mu (du_i/dx_j + du_j/dx_i - 2/3 delta_ij theta),
//   Omega = < |curl u|^2 >,
// averaged with the cell volumes over the box (the weights of the bulk integrals,
// src/calc_stress.cu:162-201). The gradients are those of derVelX/Y/Z at the viscous order
// (src/calc_stress.cu:20-63, with the velocity ghosts of src/boundary_condition_x.h:23-45
// and _z.h), mu that of calcState (src/cuda_main.cu:218-242). The reference has no such
// diagnostic (its dissipation is left to post-processing); for the Taylor-Green vortex eps
// is the kinetic-energy decay rate -dK/dt up to pressure-dilatation work. Computed in FP64
// from the FP64 state in both precision modes. Deterministic: per-block partials in fixed
// slots, summed in a fixed order.
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>

#include "../../include/cns.h"
#include "cns_internal.h"
#include "kernels_point.cuh"
#include "solver_internal.h"

using namespace cns;

namespace {

constexpr int DG_THREADS = 128;   // 32 x 4 points of a plane per block
constexpr int DG_NZ = 8;          // planes per block
constexpr int DG_FINAL = 512;

// warp maximum of the three magnitudes' codes into the slots, where it exceeds them
__device__ __forceinline__ void vel_track(unsigned* slots, unsigned u, unsigned v, unsigned w) {
    const unsigned mask = __activemask();
    const unsigned f[3] = {u, v, w};
    const bool first = (threadIdx.x & 31) == __ffs(mask) - 1;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (!__any_sync(mask, f[q] > __ldcg(slots + q))) continue;
        const unsigned m = __reduce_max_sync(mask, f[q]);
        if (first) atomicMax(slots + q, m);
    }
}

// the velocity ghost layer of the FP64 state (in FP32-RHS mode the ghost kernel fills the
// FP32 stencil copies, not the state), and the largest codes of the three components with it
__global__ void __launch_bounds__(256) k_ghost_vel(Geom g, Phys ph, double* u, double* v, double* w,
                                                   const double* scal, unsigned* vmax) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= ghost_count(g)) return;
    const long long c = ghost_vel_cell(g, ph, u, v, w, scal, t);
    vel_track(vmax, fx_code(u[c]), fx_code(v[c]), fx_code(w[c]));
}
__global__ void __launch_bounds__(256) k_vel_max(Geom g, const double* __restrict__ u, const double* __restrict__ v,
                                                 const double* __restrict__ w, unsigned* vmax) {
    const unsigned n = (unsigned)g.mx * (unsigned)g.my * (unsigned)g.mz, mx = (unsigned)g.mx, my = (unsigned)g.my;
    unsigned m[3] = {0, 0, 0};
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const unsigned jk = t / mx, k = jk / my;
        const long long c = g.at((int)(t - jk * mx), (int)(jk - k * my), (int)k);
        m[0] = max(m[0], fx_code(u[c]));
        m[1] = max(m[1], fx_code(v[c]));
        m[2] = max(m[2], fx_code(w[c]));
    }
    vel_track(vmax, m[0], m[1], m[2]);
}

// The nine gradients as fixed-point sums (fx.cuh; vmax: the components' largest codes, ghosts
// included; b: inverse spacings over the weights' denominator), the rest in FP64. With theta
// the trace, sum tau_ab G_ab = 2 sum G_aa^2 + sum_{a<b} (G_ab + G_ba)^2 - 2/3 theta^2.
// (Channel 128x160x192: 72 FP64 instructions of the gradients and 27 + 28 of the contraction
// and the viscosity power per point made the call 1.38 ms, this form 0.56 ms; what it spends now
// is 72 conversions to fixed point a point, every neighbour's anew, and the contraction in FP64.)
template <int V>
__global__ void __launch_bounds__(DG_THREADS, 4) k_dissip(Geom g, Phys ph, const double* __restrict__ xp, double bx,
                                                       double by, double bz, const unsigned* __restrict__ vmax,
                                                       StateIn q, double* __restrict__ part) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const int j = blockIdx.y * 4 + (threadIdx.x >> 5);
    const int k0 = blockIdx.z * DG_NZ, k1 = min(k0 + DG_NZ, g.mz);
    double phi = 0.0, ens = 0.0;
    if (i < g.mx && j < g.my) {
        int e[3];
        bool ok = true;
#pragma unroll
        for (int n = 0; n < 3; n++) {
            e[n] = fx_exponent(vmax[n]);
            ok = ok && fx_valid(vmax[n]);
        }
        const double b[3] = {g.nonuniform_x ? bx * xp[i] : bx, by, bz};
        const double* F[3] = {q.u, q.v, q.w};
        const auto column = [&](auto fixed) {
            for (int k = k0; k < k1; k++) {
                const long long c = g.at(i, j, k);
                const long long st[3] = {1, g.P, g.PS};
                double G[9];   // G[3 d + n] = d u_n / d x_d (derVelX/Y/Z)
#pragma unroll
                for (int d = 0; d < 3; d++) {
#pragma unroll
                    for (int n = 0; n < 3; n++) {
                        const double* f = F[n];
                        if constexpr (decltype(fixed)::value) {
                            FxSum s;
#pragma unroll
                            for (int l = 1; l <= V; l++)
                                s.add(fx_from(f[c + l * st[d]], e[n]) - fx_from(f[c - l * st[d]], e[n]), fxw1(V, l));
                            G[3 * d + n] = (double)s.value() * (b[d] * fx_pow2(e[n] - 62));
                        } else {
                            double s = 0.0;
#pragma unroll
                            for (int l = 1; l <= V; l++)
                                s = fma((double)fxw1(V, l), f[c + l * st[d]] - f[c - l * st[d]], s);
                            G[3 * d + n] = s * (b[d] * 0x1p-32);
                        }
                    }
                }
                const double rr = q.r[c], uu = q.u[c], vv = q.v[c], ww = q.w[c], ee = q.e[c];
                const double en = ee * rcp_nr(rr) - 0.5 * (uu * uu + vv * vv + ww * ww);
                const double T = ph.cvInv * en;
                const double mu = (ph.vexp_is_one ? T : pow_visc(T, ph.vexp)) * ph.invRe;
                const double th = G[0] + G[4] + G[8];
                const double a = G[1] + G[3], bb = G[2] + G[6], cc = G[5] + G[7];
                const double wx = G[5] - G[7], wy = G[6] - G[2], wz = G[1] - G[3];
                double s = fma(2.0, fma(G[0], G[0], fma(G[4], G[4], G[8] * G[8])), fma(a, a, fma(bb, bb, cc * cc)));
                s = fma(-(2.0 / 3.0) * th, th, s);
                phi = fma(mu, s, phi);
                ens += fma(wx, wx, fma(wy, wy, wz * wz));
            }
        };
        if (ok) column(std::true_type());
        else column(std::false_type());   // out of the format's range (fx_valid): FP64 gradients
        const double wv = g.wvol[i];
        phi *= wv;
        ens *= wv;
    }
    __shared__ double sh[2][DG_THREADS];
    sh[0][threadIdx.x] = phi;
    sh[1][threadIdx.x] = ens;
    __syncthreads();
    for (int h = DG_THREADS / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            sh[0][threadIdx.x] += sh[0][threadIdx.x + h];
            sh[1][threadIdx.x] += sh[1][threadIdx.x + h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const long long bl = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        part[2 * bl] = sh[0][0];
        part[2 * bl + 1] = sh[1][0];
    }
}

// the block partials summed in a fixed order: thread t takes partials t, t + DG_FINAL, ..., then a
// fixed tree; the means over the box volume
__global__ void __launch_bounds__(DG_FINAL) k_dissip_final(const double* __restrict__ part, long long nb, double vol,
                                                           double* __restrict__ out) {
    double a = 0.0, b = 0.0;
    for (long long t = threadIdx.x; t < nb; t += DG_FINAL) {
        a += part[2 * t];
        b += part[2 * t + 1];
    }
    __shared__ double sh[2][DG_FINAL];
    sh[0][threadIdx.x] = a;
    sh[1][threadIdx.x] = b;
    __syncthreads();
    for (int h = DG_FINAL / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            sh[0][threadIdx.x] += sh[0][threadIdx.x + h];
            sh[1][threadIdx.x] += sh[1][threadIdx.x + h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = sh[0][0] / vol;
        out[1] = sh[1][0] / vol;
    }
}

int diag_error(cudaError_t e) {
    return cns::set_error(e == cudaErrorMemoryAllocation ? CNS_ERR_OOM : CNS_ERR_CUDA, cudaGetErrorString(e));
}

}  // namespace

extern "C" {

int cns_dissipation(cns_solver* h, double* out) {
    if (!h || !out) return cns::set_error(CNS_ERR_INVALID, "NULL argument");
    if (!h->initialized) return cns::set_error(CNS_ERR_STATE, "no field has been copied in");
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return diag_error(e);
    const Geom& g = h->geom;
    const int c = h->cur;
    const StateIn q{h->q[c][0], h->q[c][1], h->q[c][2], h->q[c][3], h->q[c][4]};
    const dim3 grid((g.mx + 31) / 32, (g.my + 3) / 4, (g.mz + DG_NZ - 1) / DG_NZ);
    const long long nb = (long long)grid.x * grid.y * grid.z;
    double* buf = nullptr;   // partials, the two means, the largest codes
    if (cns::solver_scratch(h, 2 * (size_t)nb + 4, &buf)) return CNS_ERR_OOM;
    unsigned* vmax = (unsigned*)(buf + 2 * nb + 2);
    e = cudaMemsetAsync(vmax, 0, 4 * sizeof(unsigned), h->stream);
    if (e != cudaSuccess) return diag_error(e);
    const unsigned gb = (unsigned)((ghost_count(g) + 255) / 256);
    k_ghost_vel<<<gb, 256, 0, h->stream>>>(g, h->phys, h->q[c][1], h->q[c][2], h->q[c][3], h->scal, vmax);
    k_vel_max<<<4 * GB300_SMS, 256, 0, h->stream>>>(g, h->q[c][1], h->q[c][2], h->q[c][3], vmax);
    const int V = h->p.stencil_visc;
    const double s = ldexp(1.0, 32 - fxs1(V)) / fxn1(V), bx = g.dx * s, by = g.dy * s, bz = g.dz * s;
#define CNS_DISSIP(VV) k_dissip<VV><<<grid, DG_THREADS, 0, h->stream>>>(g, h->phys, h->xp_d, bx, by, bz, vmax, q, buf)
    switch (V) {
    case 1: CNS_DISSIP(1); break;
    case 2: CNS_DISSIP(2); break;
    case 3: CNS_DISSIP(3); break;
    default: CNS_DISSIP(4); break;
    }
#undef CNS_DISSIP
    const double vol = h->phys.Lx * h->phys.Ly * h->phys.Lz;
    k_dissip_final<<<1, DG_FINAL, 0, h->stream>>>(buf, nb, vol, buf + 2 * nb);
    h->launches += 4;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, buf + 2 * nb, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    return e == cudaSuccess ? CNS_OK : diag_error(e);
}

}  // extern "C"
