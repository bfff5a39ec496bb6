// kernels_common.cu -- state recovery, ghost fills, fixed-point conversion, dilatation,
// reductions and layout conversion. The RHS/stage kernel lives in kernels_rhs.cuh.
#include "cns_common.cuh"
#include "cns_internal.h"
#include "kernels_fx.cuh"
#include "kernels_point.cuh"

namespace cns {

// Single-solver kernels: thin grids over the per-point bodies of kernels_point.cuh.
template <typename R>
__global__ void __launch_bounds__(128) k_state(Geom g, Phys ph, StateIn q, DerivedOut<R> o, double* scal,
                                               int adv, double* time_log, long long tcap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (adv && i == 0 && j == 0 && k == 0) advance_time(scal, time_log, tcap);
    if (i >= g.mx || j >= g.my) return;
    state_point<R>(g, ph, q, o, scal, i, j, k);
}

// the time advance of stage 0 of a step when the state recovery is fused into the RHS
__global__ void k_advance_time(double* scal, double* time_log, long long tcap) {
    if (threadIdx.x == 0 && blockIdx.x == 0) advance_time(scal, time_log, tcap);
}

// adv: the first stage of a step also advances the time here, unless the ghosts depend on it
// (wall perturbation): one launch fewer per step
template <typename R>
__global__ void __launch_bounds__(256) k_ghost_state(Geom g, Phys ph, StencilFields<R> f, double* scal, int adv,
                                                     double* time_log, long long tcap) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (adv && t == 0) advance_time(scal, time_log, tcap);
    if (t < ghost_count(g)) ghost_state_cell<R>(g, ph, f, scal, t);
}

// FP32-RHS dilatation from the packed records (rho, u, v, w), marching in z: blocks of
// 32 x 8 threads, DIL_NZ (8) planes each (dil_column_packed, kernels_point.cuh).
constexpr int DIL_TX = 32, DIL_TY = 8, DIL_NZ = 8;

template <int V>
__global__ void __launch_bounds__(DIL_TX * DIL_TY) k_dil_march(Geom g, CoefT<float> cf, const float4* __restrict__ qa,
                                                               float* __restrict__ dil, int own, int nz) {
    __shared__ float su[DIL_TY][DIL_TX + 2 * V];   // u of the tile rows, x halo V on each side
    __shared__ float sv[DIL_TY + 2 * V][DIL_TX];   // v of the tile columns, y halo V on each side
    const int k0 = blockIdx.z * nz;
    dil_column_packed<V, DIL_TY, true>(g, cf, qa, dil, blockIdx.x * DIL_TX, blockIdx.y * DIL_TY, k0,
                                 min(k0 + nz, g.mz), own != 0, (int)threadIdx.x, (int)threadIdx.y, su, sv);
}

// FP64 mode: fixed-point conversion and theta. Blocks of 32 x 8 threads: the first ones write
// the stage's scale factors (16^3 box: by one block beside its tile 14 us for the kernel, so
// 9.9), the next `tiles` march nz planes of a 32 x 8 tile each (fx_column), the others convert
// 256 ghost cells each.
constexpr int FX_TABLE_BLOCKS = (FXK_COUNT + DIL_TY - 1) / DIL_TY;
template <int V>
__global__ void __launch_bounds__(DIL_TX * DIL_TY, 4) k_fx(const __grid_constant__ Geom g,
                                                           const __grid_constant__ CoefT<double> cf,
                                                           const __grid_constant__ RhsIn<double> in, int own, int tiles,
                                                           int nbx, int nby, int nz) {
    __shared__ i64 su[DIL_TY][DIL_TX + 2 * V];   // u of the tile rows, x halo V on each side
    __shared__ i64 sv[DIL_TY + 2 * V][DIL_TX];   // v of the tile columns, y halo V on each side
    __shared__ unsigned sl[2];
    const int tid = threadIdx.y * DIL_TX + threadIdx.x;
    const unsigned seen = tid < 2 ? __ldcg(in.fx.gnext + FX_LEAST + tid) : 0u;
    int e[8];
    const bool wide = !fx_exponents(cf.fx, in.fx.gmax, e);
    int t = (int)blockIdx.x - FX_TABLE_BLOCKS;
    if (t < 0) {   // an entry per warp: the entries' branches differ, one warp would take them in turn
        const int q = blockIdx.x * DIL_TY + threadIdx.y;
        if (threadIdx.x == 0 && q < FXK_COUNT) in.fx.k[q] = fx_table(cf.fx, in.fx.gmax, cf.lam_mu, q);
        return;
    }
    if (t >= tiles) {
        t = (t - tiles) * DIL_TX * DIL_TY + tid;
        FxLeast least;
        if (t < ghost_count(g)) fx_ghost(g, in, e, t, wide, least);
        least.raise_block(in.fx.gnext, sl, tid, seen);
        return;
    }
    const int r = t / nbx, bz = r / nby, k0 = bz * nz;
    const int i0 = (t - r * nbx) * DIL_TX, j0 = (r - bz * nby) * DIL_TY, k1 = min(k0 + nz, g.mz);
    FxLeast least;
    if (wide) {
        const int i = i0 + (int)threadIdx.x, j = j0 + (int)threadIdx.y;
        if (i < g.mx && j < g.my)
            for (int k = k0; k < k1; k++) {
                const int c = (int)g.at(i, j, k);
                wide_theta<V, true>(g, cf, in, i, j, k, own != 0);
                least.add(in.r[c], in.t[c]);
            }
    } else {
        fx_column<V, DIL_TY>(g, cf.fx, in, e, cf.xp, i0, j0, k0, k1, own != 0, (int)threadIdx.x, (int)threadIdx.y, su, sv,
                             least);
    }
    least.raise_block(in.fx.gnext, sl, tid, seen);
}

__global__ void __launch_bounds__(256) k_ghost_theta(Geom g, float* th) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t < ghost_count(g)) ghost_scalar_cell<float>(g, th, t);
}
__global__ void __launch_bounds__(256) k_ghost_theta(Geom g, FxFields fx) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= ghost_count(g)) return;
    if (fx.k[FXK_WIDE] == 0) ghost_scalar_cell<i64>(g, fx.th, t);
    else ghost_scalar_cell<double>(g, (double*)fx.th, t);
}

// ---------------------------------------------------------------------------------
// Reductions (deterministic two-pass: fixed partial slots, fixed summation order).
//   min dt (deviceCalcDt + minOfThreads, src/calc_stress.cu:140-160, cuda_math.cu:232-259)
//   sum rho dV, sum rho w dV, sum rhoE dV (integrateThreads, cuda_math.cu:143-171)
//   sum |u|^2 dV / V (AverageThreads, cuda_math.cu:173-201)
// partial layout: part[q*RED_BLOCKS + block], q = 1 rho, 2 rho w, 3 rhoE, 4 |u|^2,
// 5 rho |u|^2; part[RED_PEAK] the largest rate (the bit pattern of a double >= 0, zero between
// reductions)
//
// The time step is cfl over the largest of the points' convective and viscous rates (division
// rounds monotonically, so this is the smallest quotient). A rate takes three divisions and a
// square root, ~60 FP64 instructions; an FP32 estimate of it, within 1e-5 where the internal
// energy is no small difference, rules out the points that cannot exceed the largest rate found
// so far, in any block, and few are evaluated in FP64 (channel 128x160x192, a one-step run
// with its reduction and synchronisation: 0.58 -> 0.27 ms beyond the step). Each warp raises the
// largest rate once: where a thread has one point every rate exceeds the zero it starts from, and
// an atomic per point serialises at the one address (a one-step run of 77x60x41 230 -> 167 us, FP32).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

template <typename R>
__global__ void __launch_bounds__(RED_THREADS) k_reduce_partial(Geom g, Phys ph, StateIn q, const R* __restrict__ mu,
                                                                int mstride, double* part, int want) {
    __shared__ double sh[6][RED_THREADS / 32];
    const long long n = (long long)g.mx * g.my * g.mz;
    unsigned long long* peak = (unsigned long long*)(part + RED_PEAK);
    double s_r = 0.0, s_rw = 0.0, s_e = 0.0, s_k = 0.0, s_rk = 0.0;
    const float gg = (float)(ph.gam * (ph.gam - 1)), fdy = (float)g.dy, fdz = (float)g.dz,
                fd2 = fmaxf((float)g.d2y, (float)g.d2z);
    // 32-bit index arithmetic: n is below the padded field size, itself below 2^31
    const unsigned mx = (unsigned)g.mx, my = (unsigned)g.my;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const unsigned tt = (unsigned)t, jk = tt / mx;
        const int i = (int)(tt - jk * mx);
        const int j = (int)(jk % my);
        const int k = (int)(jk / my);
        const long long c = g.at(i, j, k);
        const double rr = q.r[c], uu = q.u[c], vv = q.v[c], ww = q.w[c], ee = q.e[c];
        const double wv = g.wvol[i];
        if (want & RED_DT) {
            const double found = __longlong_as_double((long long)__ldcg(peak));
            const double dx = g.dxv[i];
            const R mr = mu[c * mstride];
            const float r = d2f(rr), u = d2f(uu), v = d2f(vv), w = d2f(ww), fx = 1.0f / d2f(dx);
            const float er = d2f(ee) / r, ien = er - 0.5f * (u * u + v * v + w * w), a = sqrtf(gg * ien);
            const float m = sizeof(R) == 4 ? (float)mr : d2f((double)mr);
            const float est = fmaxf(fmaxf((fabsf(u) + a) * fx, fmaxf((fabsf(v) + a) * fdy, (fabsf(w) + a) * fdz)),
                                    m * fmaxf(fx * fx, fd2));
            // (NaN, infinity and anything below the FP32 range fail the comparisons)
            if (!(est * 1.00001f < d2f(found) * 0.999999f) || !(ien > 0.1f * er)) {
                const double en = ee / rr - 0.5 * (uu * uu + vv * vv + ww * ww);
                const double sos = sqrt(ph.gam * (ph.gam - 1) * en);
                const double d2x = dx * dx, md = to_d<R>(mr);
                const double ci = fmax((fabs(uu) + sos) / dx, fmax((fabs(vv) + sos) * g.dy, (fabs(ww) + sos) * g.dz));
                const double vi = fmax(md / d2x, fmax(md * g.d2y, md * g.d2z));
                double x = fmax(ci, vi);
                if (!(x > found)) x = 0.0;   // NaN too
                const unsigned mask = __activemask();
                const unsigned hi = __reduce_max_sync(mask, (unsigned)__double2hiint(x));
                const unsigned lo =
                    __reduce_max_sync(mask, (unsigned)__double2hiint(x) == hi ? (unsigned)__double2loint(x) : 0u);
                const unsigned long long m64 = (unsigned long long)hi << 32 | lo;
                if ((threadIdx.x & 31) == __ffs(mask) - 1 && m64 > __ldcg(peak)) atomicMax(peak, m64);
            }
        }
        if (want & RED_FORCE) { s_r += rr * wv; s_rw += rr * ww * wv; }
        if (want & RED_ENERGY) s_e += ee * wv;
        if (want & RED_KE) {
            const double q2 = (uu * uu + vv * vv + ww * ww) * wv;
            s_k += q2;
            s_rk += rr * q2;
        }
    }
    double vals[6] = {0.0, warp_sum(s_r), warp_sum(s_rw), warp_sum(s_e), warp_sum(s_k), warp_sum(s_rk)};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0)
        for (int qq = 1; qq < 6; qq++) sh[qq][wid] = vals[qq];
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0, c2 = 0, d = 0, e2 = 0, f2 = 0;
        for (int w = 0; w < RED_THREADS / 32; w++) {
            b += sh[1][w]; c2 += sh[2][w]; d += sh[3][w]; e2 += sh[4][w]; f2 += sh[5][w];
        }
        part[1 * RED_BLOCKS + blockIdx.x] = b;
        part[2 * RED_BLOCKS + blockIdx.x] = c2;
        part[3 * RED_BLOCKS + blockIdx.x] = d;
        part[4 * RED_BLOCKS + blockIdx.x] = e2;
        part[5 * RED_BLOCKS + blockIdx.x] = f2;
    }
}

// Final pass: one block. Writes dt (and dpdz with forcing, calcPressureGrad law
// src/calc_stress.cu:16-18) into the scalar block, and the bulk diagnostics into
// diag[2 s], diag[2 s + 1] (s = the device step counter) when requested:
// unforced: <u.u> (the reference's kin) and <rho |u|^2>/2; forced: bulk velocity
// int(rho w)/int(rho) and int(rhoE) (calcBulk).
__global__ void __launch_bounds__(RED_THREADS) k_reduce_final(Phys ph, double* part, int nblocks, int want,
                                                              double* scal, double* diag) {
    __shared__ double sh[6][RED_THREADS / 32];
    double b = 0, c = 0, d = 0, e = 0, f = 0;
    for (int t = threadIdx.x; t < nblocks; t += blockDim.x) {
        b += part[1 * RED_BLOCKS + t];
        c += part[2 * RED_BLOCKS + t];
        d += part[3 * RED_BLOCKS + t];
        e += part[4 * RED_BLOCKS + t];
        f += part[5 * RED_BLOCKS + t];
    }
    double vals[6] = {0.0, warp_sum(b), warp_sum(c), warp_sum(d), warp_sum(e), warp_sum(f)};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0)
        for (int q = 1; q < 6; q++) sh[q][wid] = vals[q];
    __syncthreads();
    if (threadIdx.x != 0) return;
    b = c = d = e = f = 0;
    for (int w = 0; w < RED_THREADS / 32; w++) {
        b += sh[1][w]; c += sh[2][w]; d += sh[3][w]; e += sh[4][w]; f += sh[5][w];
    }
    if (want & RED_DT) {
        scal[SC_DT] = fmin(100000.0, ph.cfl / part[RED_PEAK]);
        part[RED_PEAK] = 0.0;
        if (want & RED_FORCE) scal[SC_DPDZ] = 0.99 * scal[SC_DPDZ] - 0.5 * (c / b - 1);
    }
    if (diag) {
        double* dg = diag + 2 * (long long)scal[SC_STEP];
        const double vol = ph.Lx * ph.Ly * ph.Lz;
        if (want & RED_KE) { dg[0] = e / ph.Lx / ph.Ly / ph.Lz; dg[1] = 0.5 * f / vol; }
        else if (want & RED_FORCE) { dg[0] = c / b; dg[1] = d; }
    }
}

// ---------------------------------------------------------------------------------
// Layout conversion between the padded device layout and contiguous [k][j][i] arrays.
// ---------------------------------------------------------------------------------
template <typename T>
// (32-bit index arithmetic: the point count is below the padded field size, below 2^31)
__global__ void __launch_bounds__(256) k_unpack(Geom g, const double* __restrict__ src, T* __restrict__ dst) {
    const long long n = (long long)g.mx * g.my * g.mz;
    const unsigned mx = (unsigned)g.mx, my = (unsigned)g.my;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const unsigned tt = (unsigned)t, jk = tt / mx;
        dst[g.at((int)(tt - jk * mx), (int)(jk % my), (int)(jk / my))] = (T)src[t];
    }
}
template <typename T>
__global__ void __launch_bounds__(256) k_pack(Geom g, const T* __restrict__ src, double* __restrict__ dst) {
    const long long n = (long long)g.mx * g.my * g.mz;
    const unsigned mx = (unsigned)g.mx, my = (unsigned)g.my;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const unsigned tt = (unsigned)t, jk = tt / mx;
        const T x = src[g.at((int)(tt - jk * mx), (int)(jk % my), (int)(jk / my))];
        dst[t] = (double)x;
    }
}

// ---------------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------------
static inline dim3 point_grid(const Geom& g) { return dim3((g.mx + 31) / 32, (g.my + 3) / 4, g.mz); }
static inline dim3 point_block() { return dim3(32, 4, 1); }
static inline unsigned ghost_blocks(const Geom& g) { return (unsigned)((ghost_count(g) + 255) / 256); }

template <typename R>
void launch_state(const Geom& g, const Phys& ph, const StateIn& q, const DerivedOut<R>& o, double* scal,
                  int advance_time, double* time_log, long long tcap, cudaStream_t s) {
    k_state<R><<<point_grid(g), point_block(), 0, s>>>(g, ph, q, o, scal, advance_time, time_log, tcap);
}
void launch_advance_time(double* scal, double* time_log, long long tcap, cudaStream_t s) {
    k_advance_time<<<1, 32, 0, s>>>(scal, time_log, tcap);
}
template <typename R>
void launch_ghost_state(const Geom& g, const Phys& ph, const StencilFields<R>& f, double* scal, int adv,
                        double* time_log, long long tcap, cudaStream_t s) {
    k_ghost_state<R><<<ghost_blocks(g), 256, 0, s>>>(g, ph, f, scal, adv, time_log, tcap);
}
void launch_ghost_theta(const Geom& g, float* th, cudaStream_t s) { k_ghost_theta<<<ghost_blocks(g), 256, 0, s>>>(g, th); }
void launch_ghost_theta(const Geom& g, const FxFields& fx, cudaStream_t s) {
    k_ghost_theta<<<ghost_blocks(g), 256, 0, s>>>(g, fx);
}
void launch_dil_packed(int V, const Geom& g, const CoefT<float>& cf, const float4* qa, float* dil, int own,
                       cudaStream_t s) {
    const int nbx = (g.mx + DIL_TX - 1) / DIL_TX, nby = (g.my + DIL_TY - 1) / DIL_TY;
    // Planes per block: 8, halved while the tiles would not make two blocks per SM (a plane is a
    // dependent step of a block). 16^3 9.0 -> 5.8 us, 24^3 9.8 -> 5.7, 48^3 9.7 -> 7.8, 64^3 9.8 -> 7.8. The
    // line at four blocks per SM was slower (64^3 9.3 us, 75 x 53 x 91 11.7 against 9.8: more z halos), at
    // one the same (64^3 7.9, 75 x 53 x 91 10.9).
    int nz = DIL_NZ;
    while (nz > 1 && (long long)nbx * nby * ((g.mz + nz - 1) / nz) < 2 * GB300_SMS) nz /= 2;
    const dim3 grid(nbx, nby, (g.mz + nz - 1) / nz);
    const dim3 block(DIL_TX, DIL_TY, 1);
    switch (V) {
    case 1: k_dil_march<1><<<grid, block, 0, s>>>(g, cf, qa, dil, own, nz); break;
    case 2: k_dil_march<2><<<grid, block, 0, s>>>(g, cf, qa, dil, own, nz); break;
    case 3: k_dil_march<3><<<grid, block, 0, s>>>(g, cf, qa, dil, own, nz); break;
    default: k_dil_march<4><<<grid, block, 0, s>>>(g, cf, qa, dil, own, nz); break;
    }
}
// Planes per block: 8, halved while the tiles would not fill the GPU's four blocks per SM
// (small boxes: a plane is a dependent step of a block).
void launch_fx(int V, const Geom& g, const CoefT<double>& cf, const RhsIn<double>& in, int own, cudaStream_t s) {
    const int nbx = (g.mx + DIL_TX - 1) / DIL_TX, nby = (g.my + DIL_TY - 1) / DIL_TY;
    int nz = DIL_NZ;
    while (nz > 1 && (long long)nbx * nby * ((g.mz + nz - 1) / nz) < 4 * GB300_SMS) nz /= 2;
    const int tiles = nbx * nby * ((g.mz + nz - 1) / nz);
    const unsigned grid = FX_TABLE_BLOCKS + (unsigned)tiles + ghost_blocks(g);
    const dim3 block(DIL_TX, DIL_TY, 1);
    switch (V) {
    case 1: k_fx<1><<<grid, block, 0, s>>>(g, cf, in, own, tiles, nbx, nby, nz); break;
    case 2: k_fx<2><<<grid, block, 0, s>>>(g, cf, in, own, tiles, nbx, nby, nz); break;
    case 3: k_fx<3><<<grid, block, 0, s>>>(g, cf, in, own, tiles, nbx, nby, nz); break;
    default: k_fx<4><<<grid, block, 0, s>>>(g, cf, in, own, tiles, nbx, nby, nz); break;
    }
}
template <typename R>
int launch_reduce(const Geom& g, const Phys& ph, const StateIn& q, const R* mu, int mstride, double* part, int want,
                  double* scal, double* diag, cudaStream_t s) {
    long long n = (long long)g.mx * g.my * g.mz;
    int nb = (int)((n + RED_THREADS - 1) / RED_THREADS);
    if (nb > RED_BLOCKS) nb = RED_BLOCKS;
    k_reduce_partial<R><<<nb, RED_THREADS, 0, s>>>(g, ph, q, mu, mstride, part, want);
    k_reduce_final<<<1, RED_THREADS, 0, s>>>(ph, part, nb, want, scal, diag);
    return 2;
}
template <typename T>
void launch_unpack(const Geom& g, const double* src, T* dst, cudaStream_t s) {
    k_unpack<T><<<1184, 256, 0, s>>>(g, src, dst);
}
template <typename T>
void launch_pack(const Geom& g, const T* src, double* dst, cudaStream_t s) {
    k_pack<T><<<1184, 256, 0, s>>>(g, src, dst);
}

#define CNS_INST(R)                                                                                               \
    template void launch_state<R>(const Geom&, const Phys&, const StateIn&, const DerivedOut<R>&, double*, int,   \
                                  double*, long long, cudaStream_t);                                                        \
    template void launch_ghost_state<R>(const Geom&, const Phys&, const StencilFields<R>&, double*, int, double*,  \
                                        long long, cudaStream_t);                                                \
    template int launch_reduce<R>(const Geom&, const Phys&, const StateIn&, const R*, int, double*, int, double*, \
                                  double*, cudaStream_t);                                                        \
    template void launch_unpack<R>(const Geom&, const double*, R*, cudaStream_t);                                 \
    template void launch_pack<R>(const Geom&, const R*, double*, cudaStream_t);
CNS_INST(double)
CNS_INST(float)

}  // namespace cns
