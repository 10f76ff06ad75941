// U stage launchers (k_snap_ur), all precisions.
#include "u_kernels.cuh"

namespace mdp {

template <typename T, int TJ, int SPL>
static void launch_ur(ForcePath &fp, int inum, cudaStream_t s)
{
    const int atoms = (inum + 31) & ~31, per_cta = UR_WARPS * 32 / SPL;
    const int grid = (atoms + per_cta - 1) / per_cta * UrJobs<T, TJ>::n;
    k_snap_ur<T, TJ, SPL><<<grid, UR_WARPS * 32, 0, s>>>(fp.poff.as<int>(), fp.prij.as<double4>(),
                                                         fp.pab.as<double4>(), inum,
                                                         fp.Ut.as<typename cplx<T>::type>(), fp.u_welem, fp.u_ipad);
}

// Four lanes share an atom's pairs while one warp per (tile, job) would leave
// schedulers without a warp: the walk over about 20 pairs is then what takes
// the time (FP64, 2J = 8: 128 atoms 19 -> 11 us, 2,000 atoms 24 -> 17 us; at
// 16,000 atoms the lanes' common sums make it 69 -> 72 us).
template <typename T, int TJ>
int launch_ui(const SnapModel &, ForcePath &fp, int inum, cudaStream_t s)
{
    if (tu_ensure_tables()) return -1;
    if (fp.timing) cudaEventRecord(fp.ev[1], s);
    if ((inum + 31) / 32 * UrJobs<T, TJ>::n <= 4 * num_sms()) launch_ur<T, TJ, 4>(fp, inum, s);
    else launch_ur<T, TJ, 1>(fp, inum, s);
    return 0;
}

#define MDP_INST(T, TJ) template int launch_ui<T, TJ>(const SnapModel &, ForcePath &, int, cudaStream_t);
MDP_INST(double, 4) MDP_INST(double, 6) MDP_INST(double, 8)
MDP_INST(float, 4) MDP_INST(float, 6) MDP_INST(float, 8)
#undef MDP_INST

}  // namespace mdp
