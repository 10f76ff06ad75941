// Y and energies with several element types (k_snap_y_me), FP64.
//
// Y^{e3} of every element block e3 is the sum over the element pairs (e1, e2) and
// couplings of beta' Z^{e1 e2}, with the coefficient of the element triple and
// component that each coupling case names (cpuSnapComputeYi, cpuSnap4.cpp:697-790):
// (e1 e2 e3) when j >= j1, (e3 e2 e1) when j1 > j >= j2, (e2 e3 e1) otherwise;
// P.betaY holds the multiplicities.  The energy sum_t sum_k beta(t, k) B^t_k
// takes the couplings j >= j1 of the same triple (e1 e2 e3) without the
// multiplicity, B^t = 2 sum_half Re(U^{e3*} Z^{e1 e2}) (cpuSnapComputeEi,
// cpuSnap4.cpp:250-420): a second set of sums over the same products.
//
// The jobs are those of k_snap_y, each the work of one warp (every output has one
// owner); a CTA takes one block e3 of one
// tile, and U, whose blocks of a tile do not fit in shared memory together at
// 2J = 8, is read through L1.  With a kernel of its own per quantity, each
// forming the products of every output layer, 3,456 atoms of two elements took
// 315 (Y) and 374 us (energy) at 2J = 6.
#include "y_kernels.cuh"

namespace mdp {

template <int TJ> struct YScaleMe {
    const YParams<double> &P;
    const double *cl;      // the atom element's coefficients after beta_0
    int tA, tB, tC;        // element triples of the three cases
    template <int J1, int J2, int J> __device__ __forceinline__ double get() const
    {
        constexpr int TRI = tri_index(J1, J2, J);
        return P.betaY[TRI] * cl[(J >= J1 ? tA : J >= J2 ? tB : tC) * nbispec(TJ) + P.kmap[TRI]];
    }
};

// two warps per scheduler at most: the two sets of sums take over 200 registers
// at 2J = 8 (the last warp takes the two smallest even jobs)
template <int TJ> __host__ __device__ constexpr int yme_warps() { return cmin(TJ + 1, 8); }

template <int TJ, int PAR>
__device__ __forceinline__ void yme_job(const double2 *__restrict__ Ut, const size_t bstride, const int nb, const int e3,
                                        const int job, double2 *__restrict__ dst, const YParams<double> &P,
                                        const double *__restrict__ cl, double &e)
{
    const int top = job < 0 ? yj_none<TJ>(PAR) : yj_top<TJ>(job);
    YSums<double, yacc_count<TJ>(PAR), true> a;
    a.zero();
#pragma unroll 1
    for (int e1 = 0; e1 < nb; e1++)
#pragma unroll 1
        for (int e2 = 0; e2 < nb; e2++) {
            const YScaleMe<TJ> sc{P, cl, (e1 * nb + e2) * nb + e3, (e3 * nb + e2) * nb + e1, (e2 * nb + e3) * nb + e1};
            int next = 0;
            y_couplings<double, TJ, PAR, 0, 0>(a, Ut + e1 * bstride, Ut + e2 * bstride, top, sc, e1 == e2, next, 1,
                                               ~0u);
        }
    if (job >= 0) y_finish<double, TJ, 2, TJ - PAR>(a, Ut + e3 * bstride, dst, top, e);
}

template <int TJ>
__global__ void __launch_bounds__(yme_warps<TJ>() * 32, 1)
k_snap_y_me(const double2 *__restrict__ Ut, int natoms, const __grid_constant__ YParams<double> P,
            const __grid_constant__ MeArgs A, double2 *__restrict__ Y, double *__restrict__ esum)
{
    constexpr int NU = idxu_count(TJ), NYH = yh_count(TJ), NW = yme_warps<TJ>();
    __shared__ double ered[NW][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int e3 = blockIdx.x / A.ntiles, tile = blockIdx.x - e3 * A.ntiles, atom = tile * 32 + lane;
    const double *cl = A.coeff + (size_t)(atom < natoms ? A.elem[atom] : 0) * A.ncoeffall + 1;
    const double2 *U = Ut + (size_t)tile * NU * 32 + lane;
    const size_t bs = (size_t)A.ntiles * NU * 32;
    double2 *dst = Y + ((size_t)e3 * A.ntiles + tile) * NYH * 32 + lane;
    double e = 0.0;
#pragma unroll 1
    for (int j0 = 0; j0 <= TJ; j0 += NW) yme_job<TJ, 0>(U, bs, A.nblk, e3, j0 + w <= TJ ? j0 + w : -1, dst, P, cl, e);
    yme_job<TJ, 1>(U, bs, A.nblk, e3, w < TJ ? TJ + 1 + w : -1, dst, P, cl, e);
    ered[w][lane] = e;
    __syncthreads();
    if (w == 0 && atom < natoms) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NW; k++) s += ered[k][lane];
        esum[(size_t)e3 * natoms + atom] = s;
    }
}

// eatom = beta_0 + 2 sum_e3 esum, less the bzero parts: of t = (e e e) only
// unless wselfallflag
__global__ void k_me_energy(const double *__restrict__ esum, int natoms, int tj, int nk, int bnorm,
                            const __grid_constant__ MeArgs A, double *__restrict__ eatom)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= natoms) return;
    const double *cl = A.coeff + (size_t)A.elem[i] * A.ncoeffall;
    double s = 0.0;
    for (int b = 0; b < A.nblk; b++) s += esum[(size_t)b * natoms + i];
    double e = cl[0] + 2.0 * s;
    if (A.bzero) {
        const int nb = A.nblk, nt = nb * nb * nb;
        for (int t = 0; t < nt; t++) {
            if (!A.wselfall && t % (nb * nb + nb + 1)) continue;   // (e e e) is e (nb^2 + nb + 1)
            int k = 0;
            for (int j1 = 0; j1 <= tj; j1++)
                for (int j2 = 0; j2 <= j1; j2++)
                    for (int j = j1 - j2; j <= min(tj, j1 + j2); j += 2)
                        if (j >= j1) e -= cl[1 + t * nk + k++] * (bnorm ? 1.0 : (double)(j + 1));
        }
    }
    eatom[i] = e;
}

template <int TJ>
int launch_y_me(const YParams<double> &yp, ForcePath &fp, int inum, int bnorm, const MeArgs &A, double *eatom,
                cudaStream_t s)
{
    if (tu_ensure_tables()) return -1;
    if (fp.esum.ensure(sizeof(double) * (size_t)A.nblk * inum)) return -1;
    int per_sm = 0;
    if (kernel_setup((const void *)k_snap_y_me<TJ>, yme_warps<TJ>() * 32, 0, &per_sm, "k_snap_y_me")) return -1;
    k_snap_y_me<TJ><<<A.nblk * A.ntiles, yme_warps<TJ>() * 32, 0, s>>>(fp.Ut.as<double2>(), inum, yp, A,
                                                                    fp.Y.as<double2>(), fp.esum.as<double>());
    k_me_energy<<<(inum + 127) / 128, 128, 0, s>>>(fp.esum.as<double>(), inum, TJ, nbispec(TJ), bnorm, A, eatom);
    return 0;
}

#define MDP_INST(TJ) \
    template int launch_y_me<TJ>(const YParams<double> &, ForcePath &, int, int, const MeArgs &, double *, cudaStream_t);
MDP_INST(4) MDP_INST(6) MDP_INST(8)
#undef MDP_INST

}  // namespace mdp
