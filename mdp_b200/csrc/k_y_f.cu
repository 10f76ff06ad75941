// Y + energy stage launchers (k_snap_y), float.
#include "y_kernels.cuh"

namespace mdp {

template <typename T, int TJ>
int launch_yi(const YParams<T> &yp, ForcePath &fp, int inum, double *eatom, cudaStream_t s)
{
    if (fp.timing) cudaEventRecord(fp.ev[2], s);
    return launch_y<T, TJ, false>(yp, fp, inum, eatom, nullptr, s);
}

// per-atom coefficients G [k][atom] (the surrogate's dE_i/dB_ik), 2J=4
int launch_yi_pa_f4(const SnapModel &m, ForcePath &fp, int inum, const float *G, cudaStream_t s)
{
    if (fp.timing) cudaEventRecord(fp.ev[2], s);
    return launch_y<float, 4, true>(m.yf, fp, inum, nullptr, G, s);
}

#define MDP_INST(TJ) \
    template int launch_yi<float, TJ>(const YParams<float> &, ForcePath &, int, double *, cudaStream_t);
MDP_INST(4) MDP_INST(6) MDP_INST(8)
#undef MDP_INST

}  // namespace mdp
