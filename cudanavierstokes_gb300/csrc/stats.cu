// stats.cu -- flow statistics of the current state on the device: the plane profiles over
// (y, z) of calcAvgChan and the wall friction Reynolds number of printRes
// (src/init.cpp:150-256), which the reference evaluates on the host after copying the
// fields back. Deterministic: fixed-order partial sums, no atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/cns.h"
#include "cns_internal.h"
#include "solver_internal.h"

using namespace cns;

namespace {

constexpr int ST_X = 32, ST_R = 8;   // x-indices and row lanes of a block
constexpr int ST_BLOCKS = 4 * GB300_SMS;    // blocks of a plane sum (a few per SM: a row is a dependent step)

// fixed-order sum of the row lanes' five values, valid in lane 0
__device__ __forceinline__ void lane_sum(double (&s)[5]) {
    __shared__ double sh[5][ST_R][ST_X];
    for (int f = 0; f < 5; f++) sh[f][threadIdx.y][threadIdx.x] = s[f];
    __syncthreads();
    if (threadIdx.y == 0)
        for (int f = 0; f < 5; f++) {
            s[f] = 0.0;
            for (int r = 0; r < ST_R; r++) s[f] += sh[f][r][threadIdx.x];
        }
}

// Per x-index sums over a slice of the (j, k) rows (coalesced along x): pass 0 sums rho,
// rho u, rho v, rho w, rhoE; pass 1 the squared deviations from the plane means. (Channel
// 128x160x192, the whole call: 128 blocks of 240 rows in turn 0.82 ms, 608 blocks of 25 rows
// per thread 0.19 ms; a pass 0.047 and 0.081 ms, of which HBM 0.023.)
__global__ void __launch_bounds__(ST_X * ST_R) k_plane_sum(Geom g, StateIn q, const double* __restrict__ mean,
                                                           double* __restrict__ part) {
    const int i = blockIdx.x * ST_X + threadIdx.x;
    const unsigned rows = (unsigned)g.my * (unsigned)g.mz, my = (unsigned)g.my;
    double s[5] = {0, 0, 0, 0, 0};
    if (i < g.mx) {
        double m[5] = {0, 0, 0, 0, 0};
        if (mean)
            for (int f = 0; f < 5; f++) m[f] = mean[f * g.mx + i];
        for (unsigned rr = blockIdx.y * ST_R + threadIdx.y; rr < rows; rr += gridDim.y * ST_R) {
            const unsigned k = rr / my;
            const long long c = g.at(i, (int)(rr - k * my), (int)k);
            const double r = q.r[c], u = q.u[c], v = q.v[c], w = q.w[c], e = q.e[c];
            if (!mean) {
                s[0] += r; s[1] = fma(r, u, s[1]); s[2] = fma(r, v, s[2]); s[3] = fma(r, w, s[3]); s[4] += e;
            } else {
                const double d[5] = {r - m[0], u - m[1], v - m[2], w - m[3], e - m[4]};
                for (int f = 0; f < 5; f++) s[f] = fma(d[f], d[f], s[f]);
            }
        }
    }
    lane_sum(s);
    if (i < g.mx && threadIdx.y == 0)
        for (int f = 0; f < 5; f++) part[((long long)f * gridDim.y + blockIdx.y) * g.mx + i] = s[f];
}

// Slices summed in a fixed order; pass 0 turns the sums into <rho>, <rho u>/<rho>, ...,
// <rhoE>, pass 1 into the mean squared deviations.
__global__ void __launch_bounds__(ST_X * ST_R) k_plane_final(int mx, int slices, double n, int pass,
                                                             const double* __restrict__ part,
                                                             double* __restrict__ out) {
    const int i = blockIdx.x * ST_X + threadIdx.x;
    double s[5] = {0, 0, 0, 0, 0};
    if (i < mx)
#pragma unroll 4
        for (int b = threadIdx.y; b < slices; b += ST_R)
            for (int f = 0; f < 5; f++) s[f] += part[((long long)f * slices + b) * mx + i];
    lane_sum(s);
    if (i >= mx || threadIdx.y != 0) return;
    for (int f = 0; f < 5; f++) s[f] = s[f] / n;
    if (pass == 0) {
        s[1] /= s[0]; s[2] /= s[0]; s[3] /= s[0];
    }
    for (int f = 0; f < 5; f++) out[f * mx + i] = s[f];
}

// u_tau rho_w / mu_w of each (j, k) wall column, block sums in a fixed tree order
__global__ void __launch_bounds__(256) k_friction(Geom g, const double* __restrict__ r, const double* __restrict__ w,
                                                  int S, double c1, double c2, double c3, double c4, double xp0,
                                                  double muw, double* __restrict__ part) {
    __shared__ double sh[256];
    const long long rows = (long long)g.my * g.mz;
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    double val = 0.0;
    if (t < rows) {
        const int j = (int)(t % g.my), k = (int)(t / g.my);
        // the reference mirrors the first S interior values evenly about the wall, so the
        // k-th difference pairs w(i = k) with w(i = k - 1)
        const double co[4] = {c1, c2, c3, c4};
        double d = 0.0;
        for (int kk = 1; kk <= S; kk++) d += co[kk - 1] * (w[g.at(kk, j, k)] - w[g.at(kk - 1, j, k)]);
        d *= xp0;
        const double rw = r[g.at(0, j, k)];
        val = sqrt(muw * fabs(d) / rw) * rw / muw;
    }
    sh[threadIdx.x] = val;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// one block: thread t sums partials t, t + 256, ..., then a fixed tree
__global__ void __launch_bounds__(256) k_sum_ordered(const double* __restrict__ part, int n, double scale,
                                                     double* __restrict__ out) {
    __shared__ double sh[256];
    double s = 0.0;
    for (int b = threadIdx.x; b < n; b += 256) s += part[b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0] * scale;
}

int stats_error(cudaError_t e) {
    return cns::set_error(e == cudaErrorMemoryAllocation ? CNS_ERR_OOM : CNS_ERR_CUDA, cudaGetErrorString(e));
}

}  // namespace

extern "C" {

int cns_plane_stats(cns_solver* h, double* out) {
    if (!h || !out) return cns::set_error(CNS_ERR_INVALID, "NULL argument");
    if (!h->initialized) return cns::set_error(CNS_ERR_STATE, "no field has been copied in");
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return stats_error(e);
    const int mx = h->p.mx, nbx = (mx + ST_X - 1) / ST_X;
    const long long rows = (long long)h->p.my * h->p.mz;
    const int slices = (int)std::max(1LL, std::min<long long>(ST_BLOCKS / nbx, (rows + ST_R - 1) / ST_R));
    double* buf = nullptr;   // partials, means, deviations
    const size_t np = (size_t)5 * slices * mx;
    if (solver_scratch(h, np + 10 * (size_t)mx, &buf)) return CNS_ERR_OOM;
    double* mean = buf + np;
    double* dev = mean + 5 * (size_t)mx;
    const StateIn q{h->q[h->cur][0], h->q[h->cur][1], h->q[h->cur][2], h->q[h->cur][3], h->q[h->cur][4]};
    const dim3 grid(nbx, slices), block(ST_X, ST_R);
    const double n = (double)h->p.my * h->p.mz;
    k_plane_sum<<<grid, block, 0, h->stream>>>(h->geom, q, nullptr, buf);
    k_plane_final<<<nbx, block, 0, h->stream>>>(mx, slices, n, 0, buf, mean);
    k_plane_sum<<<grid, block, 0, h->stream>>>(h->geom, q, mean, buf);
    k_plane_final<<<nbx, block, 0, h->stream>>>(mx, slices, n, 1, buf, dev);
    h->launches += 4;
    std::vector<double> hv(10 * (size_t)mx);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hv.data(), mean, hv.size() * sizeof(double), cudaMemcpyDeviceToHost,
                                              h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return stats_error(e);
    for (int i = 0; i < mx; i++) out[i] = h->hg.x[i];
    for (size_t c = 0; c < hv.size(); c++) out[(size_t)mx + c] = hv[c];
    return CNS_OK;
}

int cns_friction_reynolds(cns_solver* h, double* ret) {
    if (!h || !ret) return cns::set_error(CNS_ERR_INVALID, "NULL argument");
    if (!h->initialized) return cns::set_error(CNS_ERR_STATE, "no field has been copied in");
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return stats_error(e);
    const int S = h->p.stencil_size;
    const long long rows = (long long)h->p.my * h->p.mz;
    const int nb = (int)((rows + 255) / 256);
    double* buf = nullptr;
    if (solver_scratch(h, (size_t)nb + 1, &buf)) return CNS_ERR_OOM;
    // first-derivative weights at the advective order with 1/dx (the reference's
    // coeffF / dx, src/init.cpp:229-234), the metric x'(0)^-1 and mu_w = T_w^viscexp / Re, T_w = 1
    const double* c1 = h->hg.c1S[0];
    const double muw = std::pow(1.0, h->p.viscexp) / h->p.Re;
    k_friction<<<nb, 256, 0, h->stream>>>(h->geom, h->q[h->cur][0], h->q[h->cur][3], S, c1[1], S > 1 ? c1[2] : 0.0,
                                          S > 2 ? c1[3] : 0.0, S > 3 ? c1[4] : 0.0, h->hg.xp[0], muw, buf);
    k_sum_ordered<<<1, 256, 0, h->stream>>>(buf, nb, 1.0 / (double)rows, buf + nb);
    h->launches += 2;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(ret, buf + nb, sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    return e == cudaSuccess ? CNS_OK : stats_error(e);
}

}  // extern "C"
