// FP64 instantiations of the RHS + stage kernel of small boxes (two threads per point).
#include "kernels_rhs.cuh"

namespace cns {
int launch_rhs_split(int S, int V, const Geom& g, const CoefT<double>& cf, const RhsIn<double>& in,
                     const Update<double>& up, double* scal, int quirk, cudaStream_t s) {
    // whole warps on either part
    const int bw = g.mx <= 16 ? 16 : 32, bh = SPLIT_POINTS / bw;
    const dim3 grid((g.mx + bw - 1) / bw, (g.my + bh - 1) / bh, g.mz), block(bw, 2 * bh, 1);
    return rhs_dispatch(S, V, [&](auto s_, auto v_) {
        k_rhs_split<decltype(s_)::value, decltype(v_)::value><<<grid, block, 0, s>>>(g, cf, in, up, scal, quirk);
    });
}
}  // namespace cns
