// fx.cuh -- 64-bit fixed-point arithmetic of the FP64 mode's stencil sums.
//
// On this GPU an FP64 instruction issues to 2 lanes per SM per cycle, a 32 x 32 + 64-bit
// integer multiply-add to 32 and a 32-bit addition to ~104 (measured), so a term of a weighted
// sum (two multiply-adds and about four additions) costs a fifth of an FP64 one. A field f with |f| < 2^e over the
// whole grid, ghosts included, is held as F = f 2^(62 - e), truncated: exact wherever |f| >=
// 2^(e - 10) (an FP64 value has 53 bits, the format 62), elsewhere within 2^(e - 62), 2^-9 of
// the rounding of the field's large values. Sums and differences of fields are exact; the
// central-difference weights are rationals with a common denominator, so a weighted
// difference is exact up to one truncation at 2^-62 of its range. The field's exponent e
// comes from its maximum, which the kernels that write the field track (fx_track).
//
// Ranges. |F| < 2^62 (1 - 2^-21) (fx_exponent), so the sum or difference of two fields fits
// 63 bits and its balanced high half (below) 31 bits; every 64-bit accumulator's bound is
// noted where it is formed. Fields whose range is too wide for this take FP64 sums instead
// (fx_exponents, kernels_fx.cuh).
#pragma once
#include <cuda_runtime.h>

namespace cns {

typedef long long i64;

// ---- a value as h 2^32 + l with both halves signed: l the low word, h the high word plus
// the low word's sign ----
__device__ __forceinline__ int fx_lo(i64 v) { return (int)(unsigned)v; }
__device__ __forceinline__ int fx_word1(i64 v) { return (int)(v >> 32); }
__device__ __forceinline__ int fx_hi(i64 v) { return fx_word1(v) + (int)((unsigned)v >> 31); }

// a b + c as a carry pair of 32-bit multiply-adds: the RHS kernel of the channel 128x160x192
// executed 4,160 instructions per point with it (profiler's counter) against 5,886 with mad.wide.
__device__ __forceinline__ i64 fx_mad(int a, int b, i64 c) {
    i64 r;
    asm("{\n\t.reg .s32 l, h;\n\tmov.b64 {l, h}, %3;\n\tmad.lo.cc.s32 l, %1, %2, l;\n\t"
        "madc.hi.s32 h, %1, %2, h;\n\tmov.b64 %0, {l, h};\n\t}"
        : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

constexpr i64 FX_HALF = 0x80000000LL;   // rounds the division by 2^32

// a b / 2^64, |a|, |b| < 2^63 (1 - 2^-21): the product of the high halves plus the two cross
// products, rounded; the product of the low halves (below a quarter of the last bit) is left
// out. Within 0.75 of the last bit, unbiased (truncation would add up over a stencil's sums). The cross sum stays below 2^63 (1 - 2^-21) + 2^32.
__device__ __forceinline__ i64 fx_mul(i64 a, i64 b) {
    const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
    const i64 m = fx_mad(ah, bl, fx_mad(al, bh, FX_HALF));
    return fx_mad(ah, bh, (i64)fx_word1(m));
}

// a b / 2^62, |a b| < 2^124.6
__device__ __forceinline__ i64 fx_mul_by4(i64 a, i64 b) {
    const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
    const i64 m = fx_mad(ah, bl, fx_mad(al, bh, FX_HALF / 4));
    return (fx_mad(ah, bh, 0) << 2) + (m >> 30);
}

// magnitude bits of the high word, and the left shift that brings the largest of several
// values (the OR of their bits) to [2^61, 2^62), or by 30
__device__ __forceinline__ int fx_bits(i64 v) { return fx_word1(v) ^ (fx_word1(v) >> 31); }
__device__ __forceinline__ int fx_room(int bits) { return max(__clz(bits) - 2, 0); }

// sum of products a_k w_k / 2^32 with small-integer weights: two accumulators, the high
// halves' and the low halves'. With |a| < 2^63 and sum |w| <= 2^30.8 both stay below 2^61.8.
struct FxSum {
    i64 h, l;
    __device__ __forceinline__ FxSum() : h(0), l(FX_HALF) {}   // rounds value()
    __device__ __forceinline__ void add(i64 a, int w) {
        h = fx_mad(fx_hi(a), w, h);
        l = fx_mad(fx_lo(a), w, l);
    }
    __device__ __forceinline__ i64 value() const { return h + (i64)fx_word1(l); }
    // value() 2^s, s the room that it leaves (fx_room, below 32), filled from the low sum: a first
    // derivative's weights are multiples of 2^21, so where the fields' values are exact the whole
    // sum is, however close the neighbours are
    __device__ __forceinline__ i64 normal(int& s) const {
        const i64 r = l - FX_HALF, v = h + (i64)fx_word1(r);
        s = fx_room(fx_bits(v));
        const unsigned lo = __funnelshift_l((unsigned)r, (unsigned)v, s);
        const unsigned hi = __funnelshift_l((unsigned)v, (unsigned)(v >> 32), s);
        return (i64)((unsigned long long)hi << 32 | lo);
    }
    __device__ __forceinline__ i64 twice() const { return (h << 1) + ((l - FX_HALF / 2) >> 31); }
};

// ---- central-difference weights as integers: c1[k] = fxw1(K, k) / fxn1(K) etc., scaled by
// 2^s so that the sum of the magnitudes (both sides of a first derivative; one side and half
// the centre weight of a second one) stays below 2^30.8 ----
__host__ __device__ constexpr int fxs1(int K) { return K == 1 ? 30 : K == 2 ? 27 : K == 3 ? 25 : 21; }
__host__ __device__ constexpr int fxn1(int K) { return K == 1 ? 2 : K == 2 ? 12 : K == 3 ? 60 : 840; }
__host__ __device__ constexpr int fxw1(int K, int k) {
    return (K == 1 ? 1
            : K == 2 ? (k == 1 ? 8 : -1)
            : K == 3 ? (k == 1 ? 45 : k == 2 ? -9 : 1)
                     : (k == 1 ? 672 : k == 2 ? -168 : k == 3 ? 32 : -3)) * (1 << fxs1(K));
}
__host__ __device__ constexpr int fxs2(int K) { return K == 1 ? 29 : K == 2 ? 25 : K == 3 ? 21 : 16; }
__host__ __device__ constexpr int fxn2(int K) { return K == 1 ? 1 : K == 2 ? 12 : K == 3 ? 180 : 5040; }
__host__ __device__ constexpr int fxw2(int K, int k) {
    return (K == 1 ? (k == 0 ? -2 : 1)
            : K == 2 ? (k == 0 ? -30 : k == 1 ? 16 : -1)
            : K == 3 ? (k == 0 ? -490 : k == 1 ? 270 : k == 2 ? -27 : 2)
                     : (k == 0 ? -14350 : k == 1 ? 8064 : k == 2 ? -1008 : k == 3 ? 128 : -9)) * (1 << fxs2(K));
}

// ---- stencil inputs. RO: no thread of the launch writes them (the read-only path, which PTX
// allows for such data alone); otherwise an earlier phase of the same launch has written them
// and the loads are ordinary ones, ordered by the barrier between the phases ----
template <bool RO, typename T>
__device__ __forceinline__ T ld(const T* p) {
    if constexpr (RO) return __ldg(p);
    else return *p;
}

// ---- four values of a 32-byte record, one load or store ----
struct __align__(32) Fx4 {
    i64 x, y, z, w;
};
template <bool RO>
__device__ __forceinline__ Fx4 fx_load4(const Fx4* p) {
    if constexpr (!RO) {
        const longlong4_32a v = *reinterpret_cast<const longlong4_32a*>(p);
        return Fx4{v.x, v.y, v.z, v.w};
    }
    Fx4 r;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.x), "=l"(r.y), "=l"(r.z), "=l"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ void fx_store4(Fx4* p, i64 x, i64 y, i64 z, i64 w) {
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" : : "l"(p), "l"(x), "l"(y), "l"(z), "l"(w) : "memory");
}

// ---- exponents ----
// The exponent code E of a value is that of the power of two above it: |f| < 2^(E - 1022) (1 -
// 2^-21); 0 for values that count as zero. fx_valid: the sums serve fields of zeros and of largest
// magnitudes from 2^-300 to 2^300; others, infinities and NaN take FP64 sums.
constexpr int FX_EMAX = 300;
__device__ __forceinline__ unsigned fx_code(double x) {
    return (((unsigned)__double2hiint(x) & 0x7fffffffu) + 1u) >> 20;
}
__device__ __forceinline__ int fx_exponent(unsigned code) { return max((int)code - 1022, -FX_EMAX); }
__device__ __forceinline__ bool fx_valid(unsigned code) {
    return code == 0 || code - (1022 - FX_EMAX) <= 2 * FX_EMAX;
}

// x 2^(62 - e), |x| < 2^e, truncated towards zero, on the integer units
__device__ __forceinline__ i64 fx_from(double x, int e) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int ex = (int)((hi >> 20) & 0x7ffu);
    // the significand with its leading bit at 2^61, then right by e - (ex - 1022) >= 0
    const unsigned mh = (__funnelshift_l(lo, hi, 9) & 0x1fffffffu) | 0x20000000u;
    const unsigned ml = lo << 9;
    i64 m;
    asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(((i64)mh << 32) | (i64)ml), "r"(e - (ex - 1022)));   // 0 beyond 63
    const i64 s = (i64)((int)hi >> 31);
    return (m ^ s) - s;
}

// 2^a, a clamped to the range of normal numbers
__device__ __forceinline__ double fx_pow2(int a) {
    return __hiloint2double((min(max(a, -1022), 1023) + 1023) << 20, 0);
}

// ---- ranges of the fields: 16 slots of a state, raised by the kernels that form it. 0..7: the
// largest codes of rho, u, v, w, T, p, H, mu. 8, 9: of rho and T the largest 2048 minus the exponent
// field, which gives the smallest magnitude's; the conversion finds these for the next stage (in
// the recovery of every point they made a 64^3 box 6 % slower), the state kernel for its own state.
// 0 is an empty slot. Reads first, one request, as the slots are one address for all warps: a warp
// issues atomics only while it raises a slot, which is rare as codes are exponents alone. ----
constexpr int FX_SLOTS = 16, FX_LEAST = 8;
constexpr int FX_SPAN = 3;   // binades of rho and T (fx_exponents, kernels_fx.cuh)
__device__ __forceinline__ void fx_slots(const unsigned* slots, unsigned (&m)[8]) {
    i64 r[4];
    asm volatile("ld.global.cg.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(r[0]), "=l"(r[1]), "=l"(r[2]), "=l"(r[3]) : "l"(slots) : "memory");
#pragma unroll
    for (int q = 0; q < 4; q++) {
        m[2 * q] = (unsigned)r[q];
        m[2 * q + 1] = (unsigned)(r[q] >> 32);
    }
}
template <int N>
__device__ __forceinline__ void fx_raise(unsigned* slots, const unsigned (&h)[N]) {
    const unsigned mask = __activemask();
    unsigned cur[8];
    fx_slots(slots, cur);
    bool up = false;
#pragma unroll
    for (int q = 0; q < N; q++) up |= h[q] > cur[q];
    if (!__any_sync(mask, up)) return;
    const bool first = (threadIdx.y * blockDim.x + threadIdx.x) % 32 == __ffs(mask) - 1;
#pragma unroll
    for (int q = 0; q < N; q++) {
        const unsigned m = __reduce_max_sync(mask, h[q]);
        if (first && m > cur[q]) atomicMax(slots + q, m);
    }
}
__device__ __forceinline__ void fx_track(unsigned* slots, const double (&f)[8]) {
    unsigned h[8];
#pragma unroll
    for (int q = 0; q < 8; q++) h[q] = fx_code(f[q]);
    fx_raise(slots, h);
}
// the smallest magnitudes' high words of rho and T, over any number of points
struct FxLeast {
    unsigned r = 0x7fffffffu, t = 0x7fffffffu;
    __device__ __forceinline__ void add(double rho, double T) {
        r = min(r, (unsigned)__double2hiint(rho) & 0x7fffffffu);
        t = min(t, (unsigned)__double2hiint(T) & 0x7fffffffu);
    }
    __device__ __forceinline__ void raise(unsigned* slots) const {
        const unsigned m[2] = {2048u - (r >> 20), 2048u - (t >> 20)};
        fx_raise(slots + FX_LEAST, m);
    }
    // once per block of whole warps, called by all its threads (tid); sh: two words of it; seen: slot
    // tid as it was some time before (the read would lengthen a small box's kernel by 1 us here)
    __device__ __forceinline__ void raise_block(unsigned* slots, unsigned* sh, int tid, unsigned seen) const {
        if (tid < 2) sh[tid] = 0u;
        __syncthreads();
        const unsigned mr = __reduce_max_sync(0xffffffffu, 2048u - (r >> 20));
        const unsigned mt = __reduce_max_sync(0xffffffffu, 2048u - (t >> 20));
        if (tid % 32 < 2) atomicMax(sh + tid % 32, tid % 32 == 0 ? mr : mt);
        __syncthreads();
        if (tid < 2 && sh[tid] > seen) atomicMax(slots + FX_LEAST + tid, sh[tid]);
    }
};

}  // namespace cns
