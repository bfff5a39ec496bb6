// FP64 instantiations of the RHS + stage kernel (plain path).
#include "kernels_rhs.cuh"

namespace cns {
int launch_rhs_split(int S, int V, const Geom& g, const CoefT<double>& cf, const RhsIn<double>& in,
                     const Update<double>& up, double* scal, int quirk, cudaStream_t s);

int launch_rhs_fp64(int S, int V, const Geom& g, const Phys&, const CoefT<double>& cf, const RhsIn<double>& in,
                    const Update<double>& up, double* scal, int quirk, cudaStream_t s) {
    // two threads per point while the blocks of 32 x 4 points do not outnumber the SMs
    // (k_rhs_split)
    if ((long long)((g.mx + 31) / 32) * ((g.my + 3) / 4) * g.mz <= 152)
        return launch_rhs_split(S, V, g, cf, in, up, scal, quirk, s);
    return launch_rhs_t<double>(S, V, g, cf, in, up, scal, quirk, s);
}
}  // namespace cns
