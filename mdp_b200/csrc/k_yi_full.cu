// Y + energy of a caller's U (k_snap_yi, double): the stage entry points take
// whatever full-plane U the caller holds, so this path reads every row as
// given, where the engine's k_snap_y uses the inversion symmetry of its own U.
#include "engine.h"

#include <algorithm>

namespace mdp {

template <int TJ, bool PA>
static int launch_full(const YParams<double> &yp, const YiLayout &yl, ForcePath &fp, int inum, double *eatom,
                       const double *G, cudaStream_t s)
{
    if (tu_ensure_tables()) return -1;
    const size_t sm = yi_smem_bytes<TJ, PA>();
    int per_sm = 0;
    if (kernel_setup((const void *)k_snap_yi<TJ, PA>, YI_WARPS * 32, sm, &per_sm, "k_snap_yi")) return -1;
    const int blocks = std::min((inum + 31) / 32, num_sms() * per_sm);
    k_snap_yi<TJ, PA><<<blocks, YI_WARPS * 32, sm, s>>>(fp.Ut.as<double2>(), inum, yp, yl, fp.Y.as<double2>(), eatom,
                                                         G);
    return 0;
}

// G: per-atom coefficients [k][atom] in place of the model's (the beta form of
// the reference's Yi, cpuSnap4.cpp:601-691; yp then holds the factors of unit
// coefficients, and no energy is written), or null
int launch_yi_full(int tj, const YParams<double> &yp, const YiLayout &yl, ForcePath &fp, int inum, double *eatom,
                   const double *G, cudaStream_t s)
{
    switch (tj) {
    case 4: return G ? launch_full<4, true>(yp, yl, fp, inum, eatom, G, s) : launch_full<4, false>(yp, yl, fp, inum, eatom, G, s);
    case 6: return G ? launch_full<6, true>(yp, yl, fp, inum, eatom, G, s) : launch_full<6, false>(yp, yl, fp, inum, eatom, G, s);
    case 8: return G ? launch_full<8, true>(yp, yl, fp, inum, eatom, G, s) : launch_full<8, false>(yp, yl, fp, inum, eatom, G, s);
    }
    set_error("twojmax %d not supported", tj);
    return -1;
}

}  // namespace mdp
