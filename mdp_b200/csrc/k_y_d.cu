// Y + energy stage launchers (k_snap_y), double.
#include "y_kernels.cuh"

namespace mdp {

template <typename T, int TJ>
int launch_yi(const YParams<T> &yp, ForcePath &fp, int inum, double *eatom, cudaStream_t s)
{
    if (fp.timing) cudaEventRecord(fp.ev[2], s);
    return launch_y<T, TJ, false>(yp, fp, inum, eatom, nullptr, s);
}

// per-atom coefficients G [k][atom] (quadratic SNAP); no energy
template <int TJ> int launch_yi_pa_d(const YParams<double> &yp, ForcePath &fp, int inum, const double *G, cudaStream_t s)
{
    return launch_y<double, TJ, true>(yp, fp, inum, nullptr, G, s);
}

#define MDP_INST(TJ)                                                                                                \
    template int launch_yi<double, TJ>(const YParams<double> &, ForcePath &, int, double *, cudaStream_t);          \
    template int launch_yi_pa_d<TJ>(const YParams<double> &, ForcePath &, int, const double *, cudaStream_t);
MDP_INST(4) MDP_INST(6) MDP_INST(8)
#undef MDP_INST

}  // namespace mdp
