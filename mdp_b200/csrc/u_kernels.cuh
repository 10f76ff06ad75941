// U stage of the engine and the batched fit (k_snap_ur): U_i = sum_j sfac(r_ij)
// U(r_ij) + wself, mirrored to the full plane (cpuSnap4.cpp:11-244).
//
// Lane = atom (or one of its pair subsets); each lane walks its atom's pairs
// and keeps the sums in registers.  The half plane is cut into jobs -- a column
// mb and a range of its layers -- whose sums fit: a warp carries one job for 32
// lanes, recomputing per pair the recursion path that reaches its column (seed
// chain and the column's rows, one row per layer), coefficient-free as in
// cf_fwd, and adds the rows of its layers; the normalisation unorm is applied
// once at the end, and the job's rows and their mirror images are written
// straight to the tile.  No shared memory, no barriers: the FP64 (FP32) pipe
// bounds it.  At 250,000 atoms, 2J = 8: FP64 3.05 ns per atom, of which its
// 2,400 FP64 instructions per pair take 2.8 at the measured FMA rate, FP32 1.42;
// adding every row into a shared-memory tile, a read and a write per pair and
// entry, took 7.58 and 4.05.
#pragma once

#include "engine.h"

namespace mdp {

// column mb, layers jlo..jhi added; top: also column TJ/2 (its single row TJ)
struct UrJob {
    int mb, jlo, jhi, top;
};
// FP64: at most 28 complex sums (112 registers); FP32: a whole column per job
template <typename T, int TJ> struct UrJobs;
template <> struct UrJobs<double, 8> {
    static constexpr int n = 7;
    static constexpr UrJob at(int k)
    {
        constexpr UrJob j[n] = {{3, 6, 8, 1}, {0, 7, 8, 0}, {1, 7, 8, 0}, {2, 7, 8, 0},
                                {0, 0, 6, 0}, {1, 2, 6, 0}, {2, 4, 6, 0}};
        return j[k];
    }
};
template <> struct UrJobs<float, 8> {
    static constexpr int n = 4;
    static constexpr UrJob at(int k)
    {
        constexpr UrJob j[n] = {{3, 6, 8, 1}, {0, 0, 8, 0}, {1, 2, 8, 0}, {2, 4, 8, 0}};
        return j[k];
    }
};
template <typename T> struct UrJobs<T, 6> {
    static constexpr int n = 3;
    static constexpr UrJob at(int k)
    {
        constexpr UrJob j[n] = {{2, 4, 6, 1}, {0, 0, 6, 0}, {1, 2, 6, 0}};
        return j[k];
    }
};
template <typename T> struct UrJobs<T, 4> {
    static constexpr int n = 2;
    static constexpr UrJob at(int k)
    {
        constexpr UrJob j[n] = {{1, 2, 4, 1}, {0, 0, 4, 0}};
        return j[k];
    }
};

// sums of row (J, mb): a middle row's right half is the mirror of its left half
__host__ __device__ constexpr int ur_len(int mb, int J) { return 2 * mb == J ? mb + 1 : J + 1; }
__host__ __device__ constexpr int ur_off(const UrJob j, int J)
{
    int n = 0;
    for (int q = j.jlo; q < J; q++) n += ur_len(j.mb, q);
    return n;
}
template <int TJ> __host__ __device__ constexpr int ur_count(const UrJob j)
{
    return ur_off(j, j.jhi + 1) + (j.top ? TJ / 2 + 1 : 0);
}

template <typename T, int TJ> struct UrState {
    T ar, ai, br, bi;
    T pr[TJ + 1], pi[TJ + 1];
};

// seed of column C + 1: row 2C + 1 of column C mirrored
template <typename T, int TJ, int C> __device__ __forceinline__ void ur_mirror(const T (&p)[TJ + 1], const T (&q)[TJ + 1], T (&r)[TJ + 1], T (&s)[TJ + 1])
{
    constexpr int J = 2 * C + 1;
    T nr[J + 1], ni[J + 1];
#pragma unroll
    for (int ma = 0; ma <= J; ma++) {
        const T sg = ((C + ma) & 1) ? T(-1) : T(1);
        nr[J - ma] = sg * p[ma];
        ni[J - ma] = -sg * q[ma];
    }
#pragma unroll
    for (int ma = 0; ma <= J; ma++) { r[ma] = nr[ma]; s[ma] = ni[ma]; }
}
template <typename T, int TJ, int MB, int C> __device__ __forceinline__ void ur_chain(UrState<T, TJ> &s)
{
    if constexpr (C < MB) {
        if constexpr (C > 0) cf_fwd<T, TJ, 2 * C, C>(s.ar, s.ai, s.br, s.bi, s.pr, s.pi);
        cf_fwd<T, TJ, 2 * C + 1, C>(s.ar, s.ai, s.br, s.bi, s.pr, s.pi);
        ur_mirror<T, TJ, C>(s.pr, s.pi, s.pr, s.pi);
        ur_chain<T, TJ, MB, C + 1>(s);
    }
}
// rows J.. of the job's column, added from layer jlo on
template <typename T, int TJ, int K, int J, int N>
__device__ __forceinline__ void ur_column(UrState<T, TJ> &s, T (&xr)[N], T (&xi)[N])
{
    constexpr UrJob jb = UrJobs<T, TJ>::at(K);
    if constexpr (J <= jb.jhi) {
        if constexpr (J > 0) cf_fwd<T, TJ, J, jb.mb>(s.ar, s.ai, s.br, s.bi, s.pr, s.pi);
        if constexpr (J >= jb.jlo) {
            constexpr int O = ur_off(jb, J);
#pragma unroll
            for (int ma = 0; ma < ur_len(jb.mb, J); ma++) { xr[O + ma] += s.pr[ma]; xi[O + ma] += s.pi[ma]; }
        }
        if constexpr (jb.top && J == TJ - 1) {
            T tr[TJ + 1], ti[TJ + 1];
            ur_mirror<T, TJ, jb.mb>(s.pr, s.pi, tr, ti);
            cf_fwd<T, TJ, TJ, TJ / 2>(s.ar, s.ai, s.br, s.bi, tr, ti);
            constexpr int O = ur_off(jb, jb.jhi + 1);
#pragma unroll
            for (int ma = 0; ma <= TJ / 2; ma++) { xr[O + ma] += tr[ma]; xi[O + ma] += ti[ma]; }
        }
        ur_column<T, TJ, K, J + 1>(s, xr, xi);
    }
}
// row (J, MB): normalised, wself on the diagonal, with its mirror image
template <typename T, int TJ, int J, int MB, int O, int N>
__device__ __forceinline__ void ur_put(const T (&xr)[N], const T (&xi)[N], typename cplx<T>::type *__restrict__ dst,
                                       const T ws)
{
    typedef typename cplx<T>::type T2;
    T2 *a = dst + (idxu_block(J) + (J + 1) * MB) * 32, *b = dst + (idxu_block(J) + (J + 1) * (J - MB) + J) * 32;
#pragma unroll
    for (int ma = 0; ma < ur_len(MB, J); ma++) {
        const T nu = unorm<T>(J, MB, ma), sg = ((ma + MB) & 1) ? T(-1) : T(1);
        T2 v = T2{nu * xr[O + ma], nu * xi[O + ma]};
        if (ma == MB) v.x += ws;
        a[ma * 32] = v;
        if (2 * MB < J || ma < MB) b[-ma * 32] = T2{sg * v.x, -sg * v.y};
    }
}
template <typename T, int TJ, int K, int J, int N>
__device__ __forceinline__ void ur_write(const T (&xr)[N], const T (&xi)[N], typename cplx<T>::type *__restrict__ dst,
                                         const T ws)
{
    constexpr UrJob jb = UrJobs<T, TJ>::at(K);
    if constexpr (J <= jb.jhi) {
        ur_put<T, TJ, J, jb.mb, ur_off(jb, J)>(xr, xi, dst, ws);
        ur_write<T, TJ, K, J + 1>(xr, xi, dst, ws);
    } else if constexpr (jb.top) {
        ur_put<T, TJ, TJ, TJ / 2, ur_off(jb, jb.jhi + 1)>(xr, xi, dst, ws);
    }
}

template <typename T, int TJ, int K, int SPL>
__device__ __forceinline__ void ur_run(const int *__restrict__ poff, const double4 *__restrict__ prij,
                                       const double4 *__restrict__ pab, const int natoms, const int i, const int sub,
                                       typename cplx<T>::type *__restrict__ Ut, const int *__restrict__ welem,
                                       const int ipad)
{
    constexpr UrJob jb = UrJobs<T, TJ>::at(K);
    constexpr int N = ur_count<TJ>(jb), NU = idxu_count(TJ);
    T xr[N], xi[N];
#pragma unroll
    for (int k = 0; k < N; k++) { xr[k] = T(0); xi[k] = T(0); }
    int p = 0, pend = 0;
    if (i < natoms) { p = poff[i] + sub; pend = poff[i + 1]; }
    double4 g = make_double4(0.0, 0.0, 0.0, 0.0);
    double sf = 0.0;
    if (p < pend) { g = pab[p]; sf = prij[p].w; }
#pragma unroll 1
    while (p < pend) {
        UrState<T, TJ> s;
        s.ar = (T)g.x; s.ai = (T)g.y; s.br = (T)g.z; s.bi = (T)g.w;
        s.pr[0] = (T)sf;   // v_0 = sfac: the recursion is linear in its root
        s.pi[0] = T(0);
        p += SPL;
        if (p < pend) { g = pab[p]; sf = prij[p].w; }
        ur_chain<T, TJ, jb.mb, 0>(s);
        ur_column<T, TJ, K, (jb.mb == 0 ? 0 : 2 * jb.mb)>(s, xr, xi);
    }
    if constexpr (SPL > 1) {
        __syncwarp();
#pragma unroll
        for (int o = 1; o < SPL; o <<= 1)
#pragma unroll
            for (int k = 0; k < N; k++) {
                xr[k] += __shfl_xor_sync(0xffffffffu, xr[k], o);
                xi[k] += __shfl_xor_sync(0xffffffffu, xi[k], o);
            }
        if (sub) return;
    }
    // wself: with welem (element blocks of virtual atoms v = b * ipad + atom)
    // only in the atom's own element block (cpuAddWself2Ui, cpuSnap4.cpp:193-244)
    T ws = T(1);
    if (welem) ws = (welem[i % ipad] == i / ipad) ? T(1) : T(0);
    ur_write<T, TJ, K, jb.jlo>(xr, xi, Ut + (size_t)(i >> 5) * NU * 32 + (i & 31), ws);
}
template <typename T, int TJ, int K, int SPL>
__device__ __forceinline__ void ur_dispatch(const int job, const int *__restrict__ poff,
                                            const double4 *__restrict__ prij, const double4 *__restrict__ pab,
                                            const int natoms, const int i, const int sub,
                                            typename cplx<T>::type *__restrict__ Ut, const int *__restrict__ welem,
                                            const int ipad)
{
    if constexpr (K < UrJobs<T, TJ>::n) {
        if (job == K) ur_run<T, TJ, K, SPL>(poff, prij, pab, natoms, i, sub, Ut, welem, ipad);
        else ur_dispatch<T, TJ, K + 1, SPL>(job, poff, prij, pab, natoms, i, sub, Ut, welem, ipad);
    }
}

// All warps of a CTA carry the same job (one loop body in the instruction
// cache); blockIdx.x = chunk * jobs + job, so that the jobs of a chunk of atoms
// run close together and its pairs come from L2 once.  SPL lanes share an
// atom's pairs (few atoms); the pad lanes of the last tile write empty sums.
constexpr int UR_WARPS = 4;
template <typename T> __host__ __device__ constexpr int ur_min_ctas() { return sizeof(T) == 8 ? 3 : 4; }
template <typename T, int TJ, int SPL>
__global__ void __launch_bounds__(UR_WARPS * 32, ur_min_ctas<T>())
k_snap_ur(const int *__restrict__ poff, const double4 *__restrict__ prij, const double4 *__restrict__ pab, int natoms,
          typename cplx<T>::type *__restrict__ Ut, const int *__restrict__ welem, int ipad)
{
    constexpr int NJ = UrJobs<T, TJ>::n, APW = 32 / SPL;
    const int chunk = blockIdx.x / NJ, job = blockIdx.x - chunk * NJ;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int a0 = (chunk * UR_WARPS + w) * APW;
    if (a0 >= ((natoms + 31) & ~31)) return;   // whole warps leave together
    ur_dispatch<T, TJ, 0, SPL>(job, poff, prij, pab, natoms, a0 + lane / SPL, lane % SPL, Ut, welem, ipad);
}

}  // namespace mdp
