// FP64 instantiations of the RHS + stage kernel (plain path).
#include "kernels_rhs.cuh"

namespace cns {
int launch_rhs_split(int S, int V, const Geom& g, const CoefT<double>& cf, const RhsIn<double>& in,
                     const Update<double>& up, double* scal, int quirk, cudaStream_t s);

int launch_rhs_fp64(int S, int V, const Geom& g, const Phys&, const CoefT<double>& cf, const RhsIn<double>& in,
                    const Update<double>& up, double* scal, int quirk, cudaStream_t s) {
    // two threads per point while the blocks of one do not outnumber the SMs (k_rhs_split)
    const PlaneTile t = plane_tile(g.mx, g.my, 128);
    if ((long long)((g.mx + t.bw - 1) / t.bw) * ((g.my + t.bh - 1) / t.bh) * g.mz <= GB300_SMS)
        return launch_rhs_split(S, V, g, cf, in, up, scal, quirk, s);
    return launch_rhs_t<double>(S, V, g, cf, in, up, scal, quirk, s);
}
}  // namespace cns
