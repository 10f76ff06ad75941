// dE/dr stage launchers (k_snap_fc, one sweep and four sums; k_snap_fr, reverse
// mode), double.
#include "f_kernels.cuh"

namespace mdp {

// Atoms from which on the one-sweep kernel is the faster one (never at 2J = 4),
// for pairs of one element type that the pair stage has made (pab).
// Its windows of 512 pairs need some rounds per SM to level out, and it stages
// each job's coefficients; ns per atom, reverse sweep against one sweep: 2J = 8
// 7.98 / 8.12 at 35,000 atoms, 7.89 / 7.21 at 64,000, 7.72 / 6.84 at 250,000;
// 2J = 6 3.89 / 3.94, 3.76 / 3.57, 3.62 / 3.31; 2J = 4 1.62 / 1.77 at 250,000.
constexpr int FC_FROM[9] = {0, 0, 0, 0, INT_MAX, 0, 49152, 0, 49152};

template <typename T, int TJ>
int launch_fi(const SnapModel &m, ForcePath &fp, int inum, int /*nm*/, cudaStream_t s)
{
    typedef typename cplx<T>::type T2;
    if (tu_ensure_tables()) return -1;
    if (fp.timing) cudaEventRecord(fp.ev[3], s);
    int per_sm = 0;
    if constexpr (FC_FROM[TJ] != INT_MAX) {
        if (inum >= FC_FROM[TJ] && fp.pab.p && !fp.fr_pcw) {
            const size_t sm = fc_smem_bytes<T, TJ>();
            if (kernel_setup((const void *)k_snap_fc<T, TJ>, FC_THREADS, sm, &per_sm, "k_snap_fc")) return -1;
            k_snap_fc<T, TJ><<<num_sms() * per_sm, FC_THREADS, sm, s>>>(
                fp.prij.as<double4>(), fp.pab.as<double4>(), fp.pinfo.as<int2>(), fp.poff.as<int>() + inum, m.geom,
                fp.Y.as<T2>(), fp.dE.as<double4>());
            return 0;
        }
    }
    const size_t sm = fr_smem_bytes<T, TJ>();
    if (kernel_setup((const void *)k_snap_fr<T, TJ>, FR_THREADS, sm, &per_sm, "k_snap_fr")) return -1;
    const int blocks = num_sms() * per_sm;
    k_snap_fr<T, TJ><<<blocks, FR_THREADS, sm, s>>>(fp.prij.as<double4>(), fp.pinfo.as<int2>(),
                                                    fp.poff.as<int>() + inum, m.geom, fp.Y.as<T2>(),
                                                    fp.dE.as<double4>(), fp.fr_pcw);
    return 0;
}

#define MDP_INST(T, TJ) template int launch_fi<T, TJ>(const SnapModel &, ForcePath &, int, int, cudaStream_t);
MDP_INST(double, 4) MDP_INST(double, 6) MDP_INST(double, 8)
#undef MDP_INST

}  // namespace mdp
