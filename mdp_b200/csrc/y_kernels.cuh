// Y and energy stage of the engine (k_snap_y): Y_i = sum_{j1 j2} beta' Z_{j1 j2 j}(U_i)
// and E_i = e0 + 2/3 sum_half w Re(U* Y) (cpuSnap4.cpp:250-421, :697-792).
//
// Lanes are the 32 atoms of a tile, whose U half plane (rows mb <= j/2) sits
// in shared memory; rows mb > j/2 are read as its mirror.  Work is split into
// jobs: one value of m' = mb - j/2 with all layers j of one parity, left half
// of the columns (ma <= j/2).  Every product u1 u2 of a coupling (J1, J2) whose
// row indices add up to m' feeds every layer J of that coupling, so a warp
// forms each product once and adds it, times a compile-time Clebsch-Gordan
// coefficient, into the layers' sums; the job's outputs stay in its registers
// while it walks the couplings.  Jobs with m' > 0 are the mirror image of the
// right half columns of -m', so all jobs of a parity run the same code.
#pragma once

#include "engine.h"

#include <algorithm>
#include <array>


namespace mdp {

// jobs: 0..TJ are the even layers' m' = 0, -1, +1, -2, +2, ..; the next TJ the
// odd layers' m' = -1/2, +1/2, -3/2, ..; top = 2 m'
template <int TJ> __host__ __device__ constexpr int yj_count() { return 2 * TJ + 1; }
template <int TJ> __host__ __device__ constexpr int yj_top(int r)
{
    if (r <= TJ) return r == 0 ? 0 : (r & 1) ? -(r + 1) : r;
    const int q = r - TJ - 1;
    return (q & 1) ? q : -(q + 1);
}
// a top that no coupling reaches (a warp without a job keeps the others' step)
template <int TJ> __host__ __device__ constexpr int yj_none(int par) { return -2 * TJ - 2 - par; }
// accumulators: left half columns ma <= J/2 of the layers of one parity
__host__ __device__ constexpr int yacc_off(int J)
{
    int n = 0;
    for (int j = J & 1; j < J; j += 2) n += j / 2 + 1;
    return n;
}
template <int TJ> __host__ __device__ constexpr int yacc_count(int par)
{
    return yacc_off(TJ - par) + (TJ - par) / 2 + 1;
}

// Warps of a tile and tiles of a CTA: one job (or half a job) per warp and
// parity, so that all warps walk the couplings together and the unrolled
// coupling code (well over 100 KB at 2J = 8, more than the instruction cache
// holds) is fetched about once per parity and CTA.  Instruction fetch is what
// bounds this kernel: the same jobs one after the other on fewer warps took
// 32.5 ns per atom at 250,000 atoms (FP64, 2J = 8) when the warps shared every
// job and 196 ns when each warp worked on a job of its own, against 16.2 ns in
// this form.  A barrier after each J1 keeps the warps in step (FP64 16.2 ns, FP32
// 8.7; without 18.0 and 9.0; one per coupling 18.6 and 9.8).  FP32 needs half the registers, so two tiles share
// a CTA and the fetched code.
template <int TJ> __host__ __device__ constexpr int y_warps() { return TJ >= 6 ? 12 : 8; }
template <typename T, int TJ> __host__ __device__ constexpr int y_tiles() { return sizeof(T) == 4 && TJ == 8 ? 2 : 1; }

// Per parity and warp: the job (255: none) and which of every `st` items of it
// the warp takes, starting with the o-th; the warps of a job shared by two meet
// in shared-memory zone `zone`.  block[g][parity]: the couplings of group g.
constexpr int Y_MAXG = 8, Y_MAXW = 12;
struct YPlan {
    unsigned char job[2][Y_MAXW], o[2][Y_MAXW], st[2][Y_MAXW], zone[2][Y_MAXW];
    unsigned block[Y_MAXG][2];
};

// Entries 0..NL-1 of row mb of layer J
template <typename T, int J, int NL>
__device__ __forceinline__ void y_load_row(const typename cplx<T>::type *__restrict__ Us, const int mb, T (&r)[NL],
                                           T (&i)[NL])
{
    typedef typename cplx<T>::type T2;
    const T2 *p = Us + (idxu_block(J) + (J + 1) * mb) * 32;
#pragma unroll
    for (int a = 0; a < NL; a++) {
        const T2 v = p[a * 32];
        r[a] = v.x;
        i[a] = v.y;
    }
}

// layers J = J1 - J2, +2, .. <= min(TJ, J1 + J2) that a coupling pair feeds
template <int TJ, int J1, int J2> struct YC {
    static constexpr int jlo = J1 - J2;
    static constexpr int jhi = J1 + J2 <= TJ ? J1 + J2 : TJ - ((J1 + J2 + TJ) & 1);
    static constexpr int nj = jhi >= jlo ? (jhi - jlo) / 2 + 1 : 0;
    static constexpr int mc = (J1 + J2) / 2;               // last column ma1 + ma2 with M <= 0
    static constexpr int n1 = cmin(J1, mc) + 1, n2 = cmin(J2, mc) + 1;   // row entries used
};

// product (ma1, ma2) = (A, M - A) times the coefficient of layers Q.., added to t
template <typename T, int TJ, int J1, int J2, int M, int A, int Q>
__device__ __forceinline__ void y_term(T (&tr)[YC<TJ, J1, J2>::nj], T (&ti)[YC<TJ, J1, J2>::nj], const T pr,
                                       const T pi)
{
    typedef YC<TJ, J1, J2> C;
    if constexpr (Q < C::nj) {
        constexpr int K = cg_block(J1, J2, C::jlo + 2 * Q) + A * (J2 + 1) + (M - A);
        const T c = cgc<T>(K);
        if constexpr (A == cmax(0, M - J2)) { tr[Q] = c * pr; ti[Q] = c * pi; }
        else { tr[Q] += c * pr; ti[Q] += c * pi; }
        y_term<T, TJ, J1, J2, M, A, Q + 1>(tr, ti, pr, pi);
    }
}
template <typename T, int TJ, int J1, int J2, int M, int A, int Q0>
__device__ __forceinline__ void y_products(T (&tr)[YC<TJ, J1, J2>::nj], T (&ti)[YC<TJ, J1, J2>::nj],
                                           const T (&ar)[YC<TJ, J1, J2>::n1], const T (&ai)[YC<TJ, J1, J2>::n1],
                                           const T (&br)[YC<TJ, J1, J2>::n2], const T (&bi)[YC<TJ, J1, J2>::n2])
{
    if constexpr (A <= cmin(M, J1)) {
        const T pr = ar[A] * br[M - A] - ai[A] * bi[M - A];
        const T pi = ar[A] * bi[M - A] + ai[A] * br[M - A];
        y_term<T, TJ, J1, J2, M, A, Q0>(tr, ti, pr, pi);
        y_products<T, TJ, J1, J2, M, A + 1, Q0>(tr, ti, ar, ai, br, bi);
    }
}
// sums of one job: the Y entries, and with EN the part of them that is the
// energy's derivative by U_J alone (see k_snap_y_me)
template <typename T, int N, bool EN = false> struct YSums {
    T r[N], i[N], er[EN ? N : 1], ei[EN ? N : 1];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int k = 0; k < N; k++) {
            r[k] = T(0); i[k] = T(0);
            if constexpr (EN) { er[k] = T(0); ei[k] = T(0); }
        }
    }
    // layer J of coupling (J1, J2): s t added to accumulator K
    template <int J1, int J2, int J, int K> __device__ __forceinline__ void add(const T s, const T tr, const T ti)
    {
        r[K] += s * tr;
        i[K] += s * ti;
        if constexpr (EN && J >= J1) {
            constexpr double w = J == J1 ? (J2 == J ? 1.0 / 3.0 : 0.5) : 1.0;   // without the multiplicity
            er[K] += T(w) * s * tr;
            ei[K] += T(w) * s * ti;
        }
    }
};
template <typename T, int TJ, int J1, int J2, int M, int Q, typename Out>
__device__ __forceinline__ void y_store(Out &out, const T (&tr)[YC<TJ, J1, J2>::nj],
                                        const T (&ti)[YC<TJ, J1, J2>::nj], const T (&sj)[YC<TJ, J1, J2>::nj])
{
    typedef YC<TJ, J1, J2> C;
    if constexpr (Q < C::nj) {
        constexpr int J = C::jlo + 2 * Q, K = yacc_off(J) + M - (J1 + J2 - J) / 2;
        out.template add<J1, J2, J, K>(sj[Q], tr[Q], ti[Q]);
        y_store<T, TJ, J1, J2, M, Q + 1>(out, tr, ti, sj);
    }
}
// columns ma1 + ma2 = M.. of one row pair; the centre column (even layers,
// m = 0) belongs to the jobs with m' <= 0
template <typename T, int TJ, int J1, int J2, int M, typename Out>
__device__ __forceinline__ void y_columns(Out &out, const T (&ar)[YC<TJ, J1, J2>::n1],
                                          const T (&ai)[YC<TJ, J1, J2>::n1], const T (&br)[YC<TJ, J1, J2>::n2],
                                          const T (&bi)[YC<TJ, J1, J2>::n2], const T (&sj)[YC<TJ, J1, J2>::nj],
                                          const int top)
{
    typedef YC<TJ, J1, J2> C;
    if constexpr (M <= C::mc) {
        constexpr int AM = J1 + J2 - 2 * M;   // |2m|
        if constexpr (AM <= C::jhi) {
            constexpr int Q0 = AM > C::jlo ? (AM - C::jlo) / 2 : 0;   // first layer with |2m| <= J
            if (AM > 0 || top <= 0) {
                T tr[C::nj], ti[C::nj];
                y_products<T, TJ, J1, J2, M, cmax(0, M - J2), Q0>(tr, ti, ar, ai, br, bi);
                y_store<T, TJ, J1, J2, M, Q0>(out, tr, ti, sj);
            }
        }
        y_columns<T, TJ, J1, J2, M + 1>(out, ar, ai, br, bi, sj, top);
    }
}
// coefficient of coupling (J1, J2, J): the model's, or times the atom's own (PA)
template <typename T, bool PA> struct YScale {
    const YParams<T> &P;
    const T *Gs;
    template <int J1, int J2, int J> __device__ __forceinline__ T get() const
    {
        constexpr int TRI = tri_index(J1, J2, J);
        T b = P.betaY[TRI];
        if constexpr (PA) b *= Gs[P.kmap[TRI] * 32];
        return b;
    }
};
template <typename T, int TJ, int J1, int J2, int Q, typename Scale>
__device__ __forceinline__ void y_scale(T (&sj)[YC<TJ, J1, J2>::nj], const int mb1, const int mb2, const Scale &sc,
                                        const bool sym)
{
    typedef YC<TJ, J1, J2> C;
    if constexpr (Q < C::nj) {
        constexpr int J = C::jlo + 2 * Q, CGB = cg_block(J1, J2, J);
        sj[Q] = sc.template get<J1, J2, J>() * cgc<T>(CGB + mb1 * (J2 + 1) + mb2);
        if (J1 == J2 && sym && mb1 != mb2) sj[Q] += sj[Q];
        y_scale<T, TJ, J1, J2, Q + 1>(sj, mb1, mb2, sc, sym);
    }
}

// the warp's share of one coupling pair (J1, J2) of a job, the J1 factor from
// U1, the J2 factor from U2.  J1 = J2 and the same U (sym): exchanging the
// factors gives the same term, so only mb1 <= mb2 is walked (twice the weight
// off the diagonal).
template <typename T, int TJ, int J1, int J2, typename Scale, typename Out>
__device__ __forceinline__ void y_block(Out &out, const typename cplx<T>::type *__restrict__ U1,
                                        const typename cplx<T>::type *__restrict__ U2, const int top,
                                        const Scale &sc, const bool sym, int &next, const int st)
{
    typedef YC<TJ, J1, J2> C;
    if constexpr (C::nj > 0) {
        const int s = (top + J1 + J2) >> 1;   // mb1 + mb2
        if (s < 0 || s > J1 + J2) return;
        const int hi = J1 == J2 && sym ? (s >> 1) : min(J1, s);
        int mb1 = max(0, s - J2) + next;
#pragma unroll 1
        for (; mb1 <= hi; mb1 += st) {
            const int mb2 = s - mb1;
            T ar[C::n1], ai[C::n1], br[C::n2], bi[C::n2], sj[C::nj];
            y_load_row<T, J1, C::n1>(U1, mb1, ar, ai);
            y_load_row<T, J2, C::n2>(U2, mb2, br, bi);
            y_scale<T, TJ, J1, J2, 0>(sj, mb1, mb2, sc, sym);
            y_columns<T, TJ, J1, J2, 0>(out, ar, ai, br, bi, sj, top);
        }
        next = mb1 - hi - 1;
    }
}

// index of coupling pair (J1, J2) among those of its parity
__host__ __device__ constexpr int y_bit(int j1, int j2)
{
    int n = 0;
    for (int a = 0; a <= j1; a++)
        for (int b = 0; b <= a; b++)
            if (((a + b) & 1) == ((j1 + j2) & 1) && (a < j1 || b < j2)) n++;
    return n;
}

// All couplings of a parity, with a barrier after each J1 that keeps the CTA's
// warps in step (every warp calls this the same number of times).
template <typename T, int TJ, int PAR, int J1, int J2, typename Scale, typename Out>
__device__ __forceinline__ void y_couplings(Out &out, const typename cplx<T>::type *__restrict__ U1,
                                            const typename cplx<T>::type *__restrict__ U2, const int top,
                                            const Scale &sc, const bool sym, int &next, const int st,
                                            const unsigned blocks)
{
    if constexpr (J1 <= TJ) {
        if constexpr (J2 <= J1) {
            if constexpr (((J1 + J2) & 1) == PAR) {
                if (blocks >> y_bit(J1, J2) & 1) y_block<T, TJ, J1, J2>(out, U1, U2, top, sc, sym, next, st);
            }
            y_couplings<T, TJ, PAR, J1, J2 + 1>(out, U1, U2, top, sc, sym, next, st, blocks);
        } else {
            if constexpr (J1 >= 3) __syncthreads();
            y_couplings<T, TJ, PAR, J1 + 1, 0>(out, U1, U2, top, sc, sym, next, st, blocks);
        }
    }
}

// a finished job's outputs to Y (half plane); with EN != 0 its energy share into
// e: sum w Re(U* Y) (EN 1), or of the energy's own sums (EN 2)
template <typename T, int TJ, int EN, int J, typename Sums>
__device__ __forceinline__ void y_finish(const Sums &a, const typename cplx<T>::type *__restrict__ Us,
                                         typename cplx<T>::type *__restrict__ dst, const int top, double &e)
{
    typedef typename cplx<T>::type T2;
    if constexpr (J >= 0) {
        if (J >= (top < 0 ? -top : top)) {
            const bool mir = top > 0;
            const int mb = (J + top) >> 1;
            const int k0 = yh_block(J) + (mir ? (J + 1) * (J - mb) + J : (J + 1) * mb);
            const int st = mir ? -32 : 32;
            T2 *row = dst + (size_t)k0 * 32;
            const T2 *us = Us + (idxu_block(J) + k0 - yh_block(J)) * 32;
#pragma unroll
            for (int ma = 0; 2 * ma <= J; ma++) {
                if (2 * ma == J && mir) continue;
                constexpr int O = yacc_off(J);
                const bool nx = mir && ((ma + mb) & 1), ny = mir && !nx;   // signs of the mirror image
                const T2 y = T2{nx ? -a.r[O + ma] : a.r[O + ma], ny ? -a.i[O + ma] : a.i[O + ma]};
                row[ma * st] = y;
                if constexpr (EN != 0) {
                    const double wgt = (top == 0 && 2 * ma == J) ? 0.5 : 1.0;
                    const T2 u = us[ma * st];
                    T2 w = y;
                    if constexpr (EN == 2) w = T2{nx ? -a.er[O + ma] : a.er[O + ma], ny ? -a.ei[O + ma] : a.ei[O + ma]};
                    e += wgt * ((double)u.x * (double)w.x + (double)u.y * (double)w.y);
                }
            }
        }
        y_finish<T, TJ, EN, J - 2>(a, Us, dst, top, e);
    }
}

// shared-memory zones of the jobs two warps share, per parity, and their offset
template <int TJ> __host__ __device__ constexpr int y_zones(int par) { return y_warps<TJ>() - (par ? TJ : TJ + 1); }
template <int TJ> __host__ __device__ constexpr int y_zone_off(int par, int zone)
{
    return par ? y_zones<TJ>(0) * yacc_count<TJ>(0) + zone * yacc_count<TJ>(1) : zone * yacc_count<TJ>(0);
}

// the warp's job of one parity; the warps of a shared job meet in its zone
template <typename T, int TJ, bool PA, int PAR>
__device__ __forceinline__ void y_job(const YPlan &plan, const unsigned blocks,
                                      const typename cplx<T>::type *__restrict__ Us,
                                      typename cplx<T>::type *__restrict__ red,
                                      typename cplx<T>::type *__restrict__ dst, const int w,
                                      const YScale<T, PA> &sc, double &e)
{
    typedef typename cplx<T>::type T2;
    constexpr int NA = yacc_count<TJ>(PAR);
    const int job = plan.job[PAR][w], o = plan.o[PAR][w], st = plan.st[PAR][w];
    const int top = job == 255 ? yj_none<TJ>(PAR) : yj_top<TJ>(job);
    YSums<T, NA> a;
    a.zero();
    int next = o;
    y_couplings<T, TJ, PAR, 0, 0>(a, Us, Us, top, sc, true, next, st, blocks);
    T2 *z = red + y_zone_off<TJ>(PAR, plan.zone[PAR][w]) * 32;
    if (o == 1)
#pragma unroll
        for (int k = 0; k < NA; k++) z[k * 32] = T2{a.r[k], a.i[k]};
    __syncthreads();
    if (job == 255 || o == 1) return;
    if (st == 2)
#pragma unroll
        for (int k = 0; k < NA; k++) {
            const T2 v = z[k * 32];
            a.r[k] += v.x;
            a.i[k] += v.y;
        }
    y_finish<T, TJ, PA ? 0 : 1, TJ - PAR>(a, Us, dst, top, e);
}

template <typename T, int TJ, bool PA> constexpr size_t y_smem_bytes()
{
    return y_tiles<T, TJ>() * (((size_t)idxu_count(TJ) + y_zone_off<TJ>(1, y_zones<TJ>(1))) * 32 * sizeof(typename cplx<T>::type) +
                               (PA ? (size_t)nbispec(TJ) * 32 * sizeof(T) : (size_t)y_warps<TJ>() * 32 * sizeof(double)));
}

// One CTA per (group, y_tiles() tiles); blockIdx.x = group * CTAs per group + ..
// Output Y in 32-atom tiles Y[tile][k][lane], k = half-plane index (the right
// halves of the middle rows, which no consumer reads, are not written).  One
// group: eatom is written.  Several groups share the couplings of every tile (few
// tiles): group g writes its partial Y to Y + g * gstride and its energy share
// to esum[g * natoms + atom], and k_y_sum adds them up.  PA: per-atom coefficients
// G[k * gpitch + atom] in place of the model's, no energy.
template <typename T, int TJ, bool PA>
__global__ void __launch_bounds__(y_tiles<T, TJ>() * y_warps<TJ>() * 32, 1)
k_snap_y(const typename cplx<T>::type *__restrict__ Ut, int natoms, const __grid_constant__ YParams<T> P,
         const __grid_constant__ YPlan plan, int ngroups, typename cplx<T>::type *__restrict__ Y, size_t gstride,
         double *__restrict__ eatom, double *__restrict__ esum, const T *__restrict__ G, int gpitch)
{
    typedef typename cplx<T>::type T2;
    constexpr int NW = y_warps<TJ>(), NT = NW * 32, NTI = y_tiles<T, TJ>();
    constexpr int NU = idxu_count(TJ), NZ = y_zone_off<TJ>(1, y_zones<TJ>(1));
    extern __shared__ __align__(16) unsigned char smraw[];
    const int lane = threadIdx.x & 31, sub = threadIdx.x / NT, t = threadIdx.x - sub * NT, w = t >> 5;
    T2 *Us = reinterpret_cast<T2 *>(smraw) + sub * (NU + NZ) * 32;
    T2 *red = Us + NU * 32;
    unsigned char *tail = smraw + NTI * (NU + NZ) * 32 * sizeof(T2);
    T *Gs = reinterpret_cast<T *>(tail) + sub * nbispec(TJ) * 32;      // [k][lane] (PA)
    double *ered = reinterpret_cast<double *>(tail) + sub * NW * 32;   // [warp][lane]
    const int ntiles = (natoms + 31) >> 5, per = (ntiles + NTI - 1) / NTI;
    const int g = blockIdx.x / per, tile = (blockIdx.x - g * per) * NTI + sub;
    const bool on = tile < ntiles;   // a CTA's last tile can be missing
    const T2 *src = Ut + (size_t)tile * NU * 32;
    for (int k = t; k < NU * 32; k += NT) Us[k] = on ? src[k] : T2{T(0), T(0)};
    if constexpr (PA) {
        for (int k = t; k < nbispec(TJ) * 32; k += NT) {
            const int a = tile * 32 + (k & 31);
            Gs[k] = (a < natoms) ? G[(size_t)(k >> 5) * gpitch + a] : T(0);
        }
    }
    __syncthreads();
    double e = 0.0;
    // a missing tile's results go where no one reads them: its own shared tile
    T2 *dst = on ? Y + g * gstride + (size_t)tile * yh_count(TJ) * 32 + lane : Us + lane;
    const YScale<T, PA> sc{P, Gs + lane};
    y_job<T, TJ, PA, 0>(plan, plan.block[g][0], Us + lane, red + lane, dst, w, sc, e);
    y_job<T, TJ, PA, 1>(plan, plan.block[g][1], Us + lane, red + lane, dst, w, sc, e);
    if constexpr (!PA) {
        ered[w * 32 + lane] = e;
        __syncthreads();
        const int atom = tile * 32 + lane;
        if (w == 0 && atom < natoms) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < NW; k++) s += ered[k * 32 + lane];
            if (ngroups == 1) eatom[atom] = P.e0 + (2.0 / 3.0) * s;
            else esum[(size_t)g * natoms + atom] = s;
        }
    }
}

// sum of the groups' partial Y and energies, in group order
template <typename T2>
__global__ void k_y_sum(const T2 *__restrict__ part, size_t n, int ngroups, T2 *__restrict__ Y,
                        const double *__restrict__ esum, int natoms, double e0, double *__restrict__ eatom)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        T2 s = part[i];
        for (int g = 1; g < ngroups; g++) {
            const T2 v = part[g * n + i];
            s.x += v.x;
            s.y += v.y;
        }
        Y[i] = s;
    }
    if (eatom && i < (size_t)natoms) {
        double s = 0.0;
        for (int g = 0; g < ngroups; g++) s += esum[(size_t)g * natoms + i];
        eatom[i] = e0 + (2.0 / 3.0) * s;
    }
}

// Host: jobs to warps and couplings to groups, by instruction count.
template <int TJ> void y_plan(YPlan &pl, int ngroups)
{
    auto columns = [](int j1, int j2, int top) {
        double c = 24.0;
        const int jhi = j1 + j2 <= TJ ? j1 + j2 : TJ - ((j1 + j2) & 1);
        for (int m = 0; 2 * m <= j1 + j2; m++) {
            const int am = j1 + j2 - 2 * m, n = cmin(j1, m) - cmax(0, m - j2) + 1;
            int q = 0;
            for (int j = j1 - j2; j <= jhi; j += 2) q += j >= am;
            if (q && (am > 0 || top <= 0)) c += 4 * n + 2 * n * q + 2 * q;
        }
        return c;
    };
    auto items = [](int j1, int j2, int top) {
        const int s = (top + j1 + j2) / 2;
        if (top + j1 + j2 < 0 || s > j1 + j2) return 0;
        return (j1 == j2 ? s / 2 : cmin(j1, s)) - cmax(0, s - j2) + 1;
    };
    constexpr int NW = y_warps<TJ>();
    for (int par = 0; par < 2; par++) {
        const int r0 = par ? TJ + 1 : 0, nj = par ? TJ : TJ + 1;
        double cost[2 * TJMAX + 1], bcost[64] = {};
        int st[2 * TJMAX + 1], nb = 0;
        for (int r = 0; r < nj; r++) { cost[r] = 0.0; st[r] = 1; }
        for (int j1 = 0; j1 <= TJ; j1++)
            for (int j2 = 0; j2 <= j1; j2++) {
                if (((j1 + j2) & 1) != par) continue;
                for (int r = 0; r < nj; r++) {
                    const int top = yj_top<TJ>(r0 + r);
                    const double c = items(j1, j2, top) * columns(j1, j2, top);
                    cost[r] += c;
                    bcost[nb] += c;
                }
                nb++;
            }
        // spare warps join the heaviest jobs
        for (int spare = NW - nj; spare > 0; spare--) {
            int best = -1;
            for (int r = 0; r < nj; r++)
                if (st[r] == 1 && (best < 0 || cost[r] > cost[best])) best = r;
            if (best < 0) break;
            st[best] = 2;
        }
        // heaviest first, each to the least loaded scheduler (warp index mod 4)
        for (int w = 0; w < Y_MAXW; w++) { pl.job[par][w] = 255; pl.o[par][w] = 0; pl.st[par][w] = 1; pl.zone[par][w] = 0; }
        double load[4] = {0, 0, 0, 0};
        bool done[2 * TJMAX + 1][2] = {};
        int zone = 0, zof[2 * TJMAX + 1];
        for (int r = 0; r < nj; r++) zof[r] = st[r] == 2 ? zone++ : 0;
        for (;;) {
            int br = -1, bo = 0;
            for (int r = 0; r < nj; r++)
                for (int o = 0; o < st[r]; o++)
                    if (!done[r][o] && (br < 0 || cost[r] / st[r] > cost[br] / st[br])) { br = r; bo = o; }
            if (br < 0) break;
            done[br][bo] = true;
            int bs = -1;
            for (int q = 0; q < 4; q++) {
                bool room = false;
                for (int w = q; w < NW; w += 4) room |= pl.job[par][w] == 255;
                if (room && (bs < 0 || load[q] < load[bs])) bs = q;
            }
            int w = bs;
            while (pl.job[par][w] != 255) w += 4;
            pl.job[par][w] = (unsigned char)(r0 + br);
            pl.o[par][w] = (unsigned char)bo;
            pl.st[par][w] = (unsigned char)st[br];
            pl.zone[par][w] = (unsigned char)zof[br];
            load[bs] += cost[br] / st[br];
        }
        // couplings: heaviest first, each to the least loaded group
        double gl[Y_MAXG] = {};
        for (int g = 0; g < Y_MAXG; g++) pl.block[g][par] = 0;
        for (int k = 0; k < nb; k++) {
            int best = 0;
            for (int b = 1; b < nb; b++)
                if (bcost[b] > bcost[best]) best = b;
            int g = 0;
            for (int h = 1; h < ngroups; h++)
                if (gl[h] < gl[g]) g = h;
            gl[g] += bcost[best];
            pl.block[g][par] |= 1u << best;
            bcost[best] = -1.0;
        }
    }
}

// Groups of ctas CTAs: as many as keep every CTA in one wave.  Splitting a
// tile's couplings over CTAs shortens the stream of instructions each has to
// fetch (FP64, 2J = 8: 128 atoms 75 us in one group, 31 us in eight; 2,000 atoms
// 96 us in one, 54 us in two, 66 us in four, which needs two waves); with more
// tiles than half the SMs it only adds partial results to sum.  At 2J = 4 the
// code is short and one group is the fastest at every size.
template <int TJ> int y_groups(int ctas, int wave)
{
    if (TJ <= 4) return 1;
    const int g = wave / ctas;
    return g < 1 ? 1 : g > Y_MAXG ? Y_MAXG : g;
}

// Y (and, without G, the energies) of the atoms from tile t0 on, nt tiles
template <typename T, int TJ, bool PA>
int launch_y_part(const YParams<T> &yp, ForcePath &fp, int inum, int t0, int nt, int wave, double *eatom, const T *G,
                  cudaStream_t s)
{
    typedef typename cplx<T>::type T2;
    constexpr int NTI = y_tiles<T, TJ>(), NT = NTI * y_warps<TJ>() * 32;
    const size_t sm = y_smem_bytes<T, TJ, PA>();
    static const std::array<YPlan, Y_MAXG> plans = [] {
        std::array<YPlan, Y_MAXG> p;
        for (int g = 0; g < Y_MAXG; g++) y_plan<TJ>(p[g], g + 1);
        return p;
    }();
    const int atoms = std::min(nt * 32, inum - t0 * 32), ctas = (nt + NTI - 1) / NTI, ng = y_groups<TJ>(ctas, wave);
    const size_t n = (size_t)nt * yh_count(TJ) * 32;
    const T2 *U = fp.Ut.as<T2>() + (size_t)t0 * idxu_count(TJ) * 32;
    T2 *Y = fp.Y.as<T2>() + (size_t)t0 * yh_count(TJ) * 32;
    if (eatom) eatom += t0 * 32;
    if (G) G += t0 * 32;
    if (ng == 1) {
        k_snap_y<T, TJ, PA><<<ctas, NT, sm, s>>>(U, atoms, yp, plans[0], 1, Y, n, eatom, nullptr, G, inum);
        return 0;
    }
    k_snap_y<T, TJ, PA><<<ctas * ng, NT, sm, s>>>(U, atoms, yp, plans[ng - 1], ng, fp.Ypart.as<T2>(), n, eatom,
                                                   fp.esum.as<double>(), G, inum);
    k_y_sum<T2><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(fp.Ypart.as<T2>(), n, ng, Y, fp.esum.as<double>(), atoms,
                                                            yp.e0, PA ? nullptr : eatom);
    count_launches(1);
    return 0;
}

// All tiles.  A last wave that is at most half full, after a few full ones, runs
// by itself with its couplings shared (a wave of one group takes 96 us at
// 2J = 8, one of two groups 54).
template <typename T, int TJ, bool PA>
int launch_y(const YParams<T> &yp, ForcePath &fp, int inum, double *eatom, const T *G, cudaStream_t s)
{
    if (tu_ensure_tables()) return -1;
    constexpr int NTI = y_tiles<T, TJ>(), NT = NTI * y_warps<TJ>() * 32;
    int per_sm = 0;
    if (kernel_setup((const void *)k_snap_y<T, TJ, PA>, NT, y_smem_bytes<T, TJ, PA>(), &per_sm, "k_snap_y")) return -1;
    const int nt = (inum + 31) / 32, wave = num_sms() * per_sm, ctas = (nt + NTI - 1) / NTI, rem = ctas % wave;
    // The groups' parts fill at most a wave's tiles (12 MB).  The room is taken at
    // the first call of any size: a smaller system can need more of it than a
    // larger one, and a buffer must not grow while a call is captured.
    if (TJ > 4 && (fp.Ypart.ensure(sizeof(typename cplx<T>::type) * wave * NTI * yh_count(TJ) * 32) ||
                   fp.esum.ensure(sizeof(double) * wave * NTI * 32)))
        return -1;
    if (TJ > 4 && ctas > wave && ctas < 16 * wave && rem > 0 && 2 * rem <= wave) {
        const int t0 = (ctas - rem) * NTI;
        if (launch_y_part<T, TJ, PA>(yp, fp, inum, 0, t0, wave, eatom, G, s)) return -1;
        count_launches(1);
        return launch_y_part<T, TJ, PA>(yp, fp, inum, t0, nt - t0, wave, eatom, G, s);
    }
    return launch_y_part<T, TJ, PA>(yp, fp, inum, 0, nt, wave, eatom, G, s);
}

}  // namespace mdp
