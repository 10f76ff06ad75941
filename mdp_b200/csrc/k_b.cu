// Per-atom bispectrum of the engine's U (k_snap_b): B_k = 2 sum_half w Re(U_j* Z_{j1 j2 j})
// (- bzero) for the triples j >= j1 (cpuSnap4.cpp:427-592).
//
// The jobs of the Y kernel (y_kernels.cuh), one warp each: a coupling (j1, j2)
// forms each product of two U entries once for all its layers j >= j1, the warp
// contracts its rows with U, and the warps' shares of the coupling's components
// meet in shared memory, one barrier per coupling.  k_snap_bi, which walks
// whole components per warp (six instructions a term, every layer its own
// products), took 105 us for 8,192 atoms at 2J = 6 in FP64 and 195 us for 250,000
// atoms at 2J = 4 in FP32; it stays for the stage entry points, whose U need not
// have the inversion symmetry.
#include "y_kernels.cuh"

namespace mdp {

template <int TJ> __host__ __device__ constexpr int b_warps() { return TJ + 1; }
constexpr int B_MAXQ = 3;   // components of a coupling pair at most (j1 = j2 = 4)

// index of triple (j1, j2, j), j >= j1, among the components
template <int TJ> __host__ __device__ constexpr int b_index(int J1, int J2, int J)
{
    int n = 0;
    for (int j1 = 0; j1 <= TJ; j1++)
        for (int j2 = 0; j2 <= j1; j2++)
            for (int j = j1 - j2; j <= cmin(TJ, j1 + j2); j += 2)
                if (j >= j1) {
                    if (j1 == J1 && j2 == J2 && j == J) return n;
                    n++;
                }
    return -1;
}
// layers of the coupling pair below J1, which carry no component
template <int TJ, int J1, int J2> __host__ __device__ constexpr int b_skip()
{
    int n = 0;
    for (int J = YC<TJ, J1, J2>::jlo; J < J1 && J <= YC<TJ, J1, J2>::jhi; J += 2) n++;
    return n;
}

struct BScale {   // Z itself
    template <int J1, int J2, int J> __device__ __forceinline__ float get() const { return 1.0f; }
};
template <typename T, int N> struct BSums {
    T r[N], i[N];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int k = 0; k < N; k++) { r[k] = T(0); i[k] = T(0); }
    }
    template <int J1, int J2, int J, int K> __device__ __forceinline__ void add(const T s, const T tr, const T ti)
    {
        if constexpr (J >= J1) {
            r[K] += s * tr;
            i[K] += s * ti;
        }
    }
};

template <typename T> struct BArgs {
    const typename cplx<T>::type *Us;   // the lane's tile column
    double *part;                       // [2][warp][B_MAXQ][32], at the lane
    int w, top[2], turn, atom, natoms, bnorm, bzero;
    double *bout;
    long bstride;
};

// the warp's share of component (J1, J2, J1 - J2 + 2Q): 2 sum w Re(U* Z) over its
// left half columns (the centre of m' = 0 counts half, the others' right halves
// are the mirror jobs')
template <typename T, int TJ, int J1, int J2, int Q, int N>
__device__ __forceinline__ void b_dots(const BArgs<T> &A, const BSums<T, N> &a, const int top, double *__restrict__ part)
{
    typedef YC<TJ, J1, J2> C;
    if constexpr (Q < C::nj) {
        constexpr int J = C::jlo + 2 * Q, O = yacc_off(J);
        double s = 0.0;
        if (J >= (top < 0 ? -top : top)) {
            const typename cplx<T>::type *u = A.Us + (idxu_block(J) + (J + 1) * ((J + top) >> 1)) * 32;
#pragma unroll
            for (int ma = 0; 2 * ma <= J; ma++) {
                if (2 * ma == J && top > 0) continue;
                const double wgt = (2 * ma == J && top == 0) ? 1.0 : 2.0;
                const auto v = u[ma * 32];
                s += wgt * ((double)v.x * (double)a.r[O + ma] + (double)v.y * (double)a.i[O + ma]);
            }
        }
        part[(Q - b_skip<TJ, J1, J2>()) * 32] = s;
        b_dots<T, TJ, J1, J2, Q + 1>(A, a, top, part);
    }
}
template <typename T, int TJ, int PAR, int J1, int J2> __device__ __forceinline__ void b_couplings(BArgs<T> &A)
{
    typedef YC<TJ, J1, J2> C;
    if constexpr (J1 <= TJ) {
        if constexpr (J2 <= J1) {
            constexpr int SK = b_skip<TJ, J1, J2>(), NQ = C::nj - SK, NW = b_warps<TJ>();
            if constexpr (((J1 + J2) & 1) == PAR && NQ > 0) {
                static_assert(NQ <= B_MAXQ && NQ <= NW, "");
                BSums<T, yacc_count<TJ>(PAR)> a;
                a.zero();
                int next = 0;
                const int top = A.top[PAR];
                y_block<T, TJ, J1, J2>(a, A.Us, A.Us, top, BScale{}, true, next, 1);
                double *part = A.part + (A.turn & 1) * NW * B_MAXQ * 32;
                b_dots<T, TJ, J1, J2, SK>(A, a, top, part + A.w * B_MAXQ * 32);
                __syncthreads();   // (two buffers: the one after next overwrites this one)
                A.turn++;
                if (A.w < NQ && A.atom < A.natoms) {
                    double b = 0.0;
#pragma unroll
                    for (int v = 0; v < NW; v++) b += part[(v * B_MAXQ + A.w) * 32];
                    const int J = C::jlo + 2 * (SK + A.w);
                    if (A.bnorm) b /= (J + 1);
                    if (A.bzero) b -= A.bnorm ? 1.0 : (double)(J + 1);
                    // a coupling pair's components are consecutive
                    A.bout[(long)(b_index<TJ>(J1, J2, C::jlo + 2 * SK) + A.w) * A.bstride + A.atom] = b;
                }
            }
            b_couplings<T, TJ, PAR, J1, J2 + 1>(A);
        } else {
            b_couplings<T, TJ, PAR, J1 + 1, 0>(A);
        }
    }
}

template <typename T, int TJ> constexpr size_t b_smem_bytes()
{
    return (size_t)idxu_count(TJ) * 32 * sizeof(typename cplx<T>::type) +
           sizeof(double) * 2 * b_warps<TJ>() * B_MAXQ * 32;
}

template <typename T, int TJ>
__global__ void __launch_bounds__(b_warps<TJ>() * 32, 1)
k_snap_b(const typename cplx<T>::type *__restrict__ Ut, int natoms, int bnorm, int bzero, double *__restrict__ bout,
         long bstride)
{
    typedef typename cplx<T>::type T2;
    constexpr int NU = idxu_count(TJ);
    extern __shared__ __align__(16) unsigned char smraw[];
    T2 *Us = reinterpret_cast<T2 *>(smraw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, tile = blockIdx.x;
    const T2 *src = Ut + (size_t)tile * NU * 32;
    for (int k = threadIdx.x; k < NU * 32; k += b_warps<TJ>() * 32) Us[k] = src[k];
    __syncthreads();
    BArgs<T> A;
    A.Us = Us + lane;
    A.part = reinterpret_cast<double *>(Us + NU * 32) + lane;
    A.w = w;
    A.top[0] = yj_top<TJ>(w);
    A.top[1] = w < TJ ? yj_top<TJ>(TJ + 1 + w) : yj_none<TJ>(1);   // its shares are zeros
    A.turn = 0;
    A.atom = tile * 32 + lane;
    A.natoms = natoms;
    A.bnorm = bnorm;
    A.bzero = bzero;
    A.bout = bout;
    A.bstride = bstride;
    b_couplings<T, TJ, 0, 0, 0>(A);
    b_couplings<T, TJ, 1, 0, 0>(A);
}

template <typename T, int TJ>
int launch_b(const ForcePath &fp, int inum, int bnorm, int bzero, double *bout, cudaStream_t s)
{
    if (tu_ensure_tables()) return -1;
    const size_t sm = b_smem_bytes<T, TJ>();
    int per_sm = 0;
    if (kernel_setup((const void *)k_snap_b<T, TJ>, b_warps<TJ>() * 32, sm, &per_sm, "k_snap_b")) return -1;
    k_snap_b<T, TJ><<<(inum + 31) / 32, b_warps<TJ>() * 32, sm, s>>>(fp.Ut.as<typename cplx<T>::type>(), inum, bnorm,
                                                                   bzero, bout, inum);
    count_launches(1);
    MDP_CUDA_TRY(cudaGetLastError());
    return 0;
}

#define MDP_INST(T, TJ) template int launch_b<T, TJ>(const ForcePath &, int, int, int, double *, cudaStream_t);
MDP_INST(double, 4) MDP_INST(double, 6) MDP_INST(double, 8) MDP_INST(float, 4)
#undef MDP_INST

}  // namespace mdp
