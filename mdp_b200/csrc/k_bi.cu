// Per-atom bispectrum launcher (k_snap_bi) on the U tiles of a caller (the stage
// entry points, whose U need not have the inversion symmetry), FP64.
#include "engine.h"

#include <algorithm>

namespace mdp {

template <int TJ>
static int launch_bi(const double2 *Ut, int natoms, int bnorm, int bzero, double *bout, long bstride,
                     cudaStream_t s)
{
    if (tu_ensure_tables()) return -1;
    const size_t sm = (size_t)idxu_count(TJ) * 32 * sizeof(double2);
    int per_sm = 0;
    if (kernel_setup((const void *)k_snap_bi<double, TJ>, BI_WARPS * 32, sm, &per_sm, "k_snap_bi")) return -1;
    const int blocks = std::min((natoms + 31) / 32, num_sms() * per_sm);
    k_snap_bi<double, TJ><<<blocks, BI_WARPS * 32, sm, s>>>(Ut, natoms, bnorm, bzero, bout, bstride);
    count_launches(1);
    MDP_CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_bi_tiles(const double2 *Ut, int natoms, int tj, int bnorm, int bzero, double *bout, long bstride,
                    cudaStream_t s)
{
    switch (tj) {
    case 4: return launch_bi<4>(Ut, natoms, bnorm, bzero, bout, bstride, s);
    case 6: return launch_bi<6>(Ut, natoms, bnorm, bzero, bout, bstride, s);
    case 8: return launch_bi<8>(Ut, natoms, bnorm, bzero, bout, bstride, s);
    }
    set_error("twojmax %d not supported", tj);
    return -1;
}

}  // namespace mdp
