// dE/dr stage (k_snap_fc): dE/d(r_j - r_i) of every pair, the force part of
// cpuSnap4.cpp:798-1175.
//
// With F(a, b) = sum_half w Re(Y* u(a, b)), dE/dx_k = 2 (dsfac e_k F + sfac dF/dx_k)
// (e = r / |r|).  (a, b) lies on the unit sphere |a|^2 + |b|^2 = 1, so its
// derivative along x_k is an infinitesimal rotation: with
//     i alpha_k = a conj(da) + conj(b) db,   beta_k = conj(b) da - a conj(db)
// a coefficient-free row v (u = unorm v, the form of cf_fwd), which is a
// homogeneous polynomial in the rotated variables, changes by
//     dv[m] = i alpha (J - 2m) v[m] + beta (J - m + 1) v[m-1] - conj(beta) (m + 1) v[m+1].
// All three directions' derivatives are therefore F's own sum with three other
// sets of coefficients, which depend on the atom only:
//     F = Re sum v C0,  Gz = dF/dalpha = -sum (J - 2m) Im(v C0),
//     Gx = dF/dRe(beta) = Re sum v Cx,  Gy = dF/dIm(beta) = Re sum v Cy,
//     C0 = conj(y),  P[m] = (J - m) conj(y[m+1]),  Q[m] = -m conj(y[m-1]),
//     Cx = P + Q,  Cy = i (P - Q),  y = w unorm Y
// and a pair needs one forward sweep of the recursion and four sums over its
// 145 entries (17 instructions an entry) instead of the forward and adjoint
// rows of a reverse-mode sweep (about 35, at twice the registers).  A middle
// row (J = 2 mb) keeps its left half and centre; the source v[mb+1] of the
// centre's term is the mirror of v[mb-1] and is folded into that entry.
//
// The half plane is cut into the jobs of the U kernel (a column, a range of its
// layers), whose loop bodies are short enough for the instruction cache.  A CTA
// takes windows of consecutive pairs and goes through the jobs: the C of one
// job's entries is staged for up to fc_cap() of the window's atoms, then every
// warp runs the job's body over the window's pairs, 32 at a time, and adds to the
// pairs' sums in shared memory.  At 250,000 atoms, 2J = 8: FP64 6.84 ns per atom
// against 7.72 of the reverse sweep, FP32 4.87 against 6.15.  One column per
// warp, all entries staged at once, left the warps of an SM in four bodies of
// 15 KB and waiting for instructions (3.7 of 11 stall cycles per instruction).
#pragma once

#include "u_kernels.cuh"

#include <climits>

namespace mdp {

template <int TJ> using FcJobs = UrJobs<double, TJ>;
constexpr int FC_THREADS = 256;
template <typename T> __host__ __device__ constexpr int fc_pairs() { return sizeof(T) == 8 ? 512 : 1024; }
// atoms staged at a time (a window at 19 pairs per atom spans 28 / 55; one of
// more takes several turns)
template <typename T> __host__ __device__ constexpr int fc_cap() { return sizeof(T) == 8 ? 30 : 58; }
template <int TJ> __host__ __device__ constexpr int fc_most()   // entries of the largest job
{
    int m = 0;
    for (int k = 0; k < FcJobs<TJ>::n; k++) m = cmax(m, ur_count<TJ>(FcJobs<TJ>::at(k)));
    return m;
}
template <int TJ> __host__ __device__ constexpr int fc_base(int job)   // entries of the jobs before
{
    int n = 0;
    for (int k = 0; k < job; k++) n += ur_count<TJ>(FcJobs<TJ>::at(k));
    return n;
}

// How an entry's coefficients come from its Y row: C0 = n0 conj(y[0]), P = (px
// Re, py Im) of y[dp], Q = nq conj(y[dq]); offsets in lanes of the Y tile
struct FcEntry {
    double n0, px, py, nq;
    int k, dp, dq;
};
template <typename T, int TJ> constexpr size_t fc_smem_bytes()
{
    return (size_t)fc_most<TJ>() * 3 * fc_cap<T>() * sizeof(typename cplx<T>::type) +
           fc_pairs<T>() * (4 * sizeof(double) + 4 * sizeof(T) + sizeof(int)) +
           fc_base<TJ>(FcJobs<TJ>::n) * sizeof(FcEntry) + sizeof(int);
}

// Y tile offsets and factors of entry m of row (J, mb)
__device__ __forceinline__ FcEntry fc_entry(const int J, const int mb, const int ma)
{
    const bool mid = 2 * mb == J;
    FcEntry c;
    c.k = (yh_block(J) + (J + 1) * mb + ma) * 32;
    c.n0 = unorm<double>(J, mb, ma) * ((mid && ma == mb) ? 0.5 : 1.0);
    const bool up = mid ? ma < mb : ma < J, down = ma > 0;
    c.dp = up ? 32 : 0;
    c.px = up ? unorm<double>(J, mb, ma + 1) * (J - ma) : 0.0;
    // left of the centre: half weight twice, the second from the mirror's source
    c.py = (mid && ma + 1 == mb) ? 0.0 : -c.px;
    c.dq = down ? -32 : 0;
    c.nq = down ? -unorm<double>(J, mb, ma - 1) * ma : 0.0;
    return c;
}
// stored as pairs (Re, -Im), so that Re(v C) is a plain dot product
template <typename T>
__device__ __forceinline__ void fc_coeffs(const FcEntry &c, const typename cplx<T>::type *__restrict__ y,
                                          typename cplx<T>::type *__restrict__ out)
{
    typedef typename cplx<T>::type T2;
    const T2 y0 = y[0], yp = y[c.dp], ym = y[c.dq];
    const T pr = (T)c.px * yp.x, pi = (T)c.py * yp.y, qr = (T)c.nq * ym.x, qi = -(T)c.nq * ym.y;
    out[0] = T2{(T)c.n0 * y0.x, (T)c.n0 * y0.y};
    out[fc_cap<T>()] = T2{pr + qr, -(pi + qi)};
    out[2 * fc_cap<T>()] = T2{qi - pi, qr - pr};   // i (P - Q) = (-(Pi - Qi), Pr - Qr)
}

// entries of the jobs, in order
template <int TJ, int K> __device__ __forceinline__ void fc_entries(FcEntry *__restrict__ ent, const int t0, const int nt)
{
    if constexpr (K < FcJobs<TJ>::n) {
        constexpr UrJob jb = FcJobs<TJ>::at(K);
        constexpr int N = ur_count<TJ>(jb), B = fc_base<TJ>(K);
        for (int q = t0; q < N; q += nt) {
            int J = jb.jlo, r = q;
            while (J <= jb.jhi && r >= ur_len(jb.mb, J)) r -= ur_len(jb.mb, J++);
            ent[B + q] = J <= jb.jhi ? fc_entry(J, jb.mb, r) : fc_entry(TJ, TJ / 2, r);
        }
        fc_entries<TJ, K + 1>(ent, t0, nt);
    }
}

// sums F, Gz, Gx, Gy over N entries of a row of layer J, C at entry offset O
template <typename T, int TJ, int J, int N, int O>
__device__ __forceinline__ void fc_dot(const T (&pr)[TJ + 1], const T (&pi)[TJ + 1],
                                       const typename cplx<T>::type *__restrict__ C,
                                       typename FAccSel<T>::type (&G)[4])
{
    typedef typename cplx<T>::type T2;
    T f = T(0), z = T(0), x = T(0), y = T(0);
#pragma unroll
    for (int m = 0; m < N; m++) {
        const T2 c0 = C[(3 * (O + m) + 0) * fc_cap<T>()], cx = C[(3 * (O + m) + 1) * fc_cap<T>()],
                 cy = C[(3 * (O + m) + 2) * fc_cap<T>()];
        f += pr[m] * c0.x + pi[m] * c0.y;
        if (J != 2 * m) z += T(J - 2 * m) * (pr[m] * c0.y - pi[m] * c0.x);
        x += pr[m] * cx.x + pi[m] * cx.y;
        y += pr[m] * cy.x + pi[m] * cy.y;
    }
    G[0].add(f);
    G[1].add(z);
    G[2].add(x);
    G[3].add(y);
}
// rows J.. of the job's column
template <typename T, int TJ, int K, int J>
__device__ __forceinline__ void fc_column(UrState<T, TJ> &s, const typename cplx<T>::type *__restrict__ C,
                                          typename FAccSel<T>::type (&G)[4])
{
    constexpr UrJob jb = FcJobs<TJ>::at(K);
    if constexpr (J <= jb.jhi) {
        if constexpr (J > 0) cf_fwd<T, TJ, J, jb.mb>(s.ar, s.ai, s.br, s.bi, s.pr, s.pi);
        if constexpr (J >= jb.jlo) fc_dot<T, TJ, J, ur_len(jb.mb, J), ur_off(jb, J)>(s.pr, s.pi, C, G);
        if constexpr (jb.top && J == TJ - 1) {
            T tr[TJ + 1], ti[TJ + 1];
            ur_mirror<T, TJ, jb.mb>(s.pr, s.pi, tr, ti);
            cf_fwd<T, TJ, TJ, TJ / 2>(s.ar, s.ai, s.br, s.bi, tr, ti);
            fc_dot<T, TJ, TJ, TJ / 2 + 1, ur_off(jb, jb.jhi + 1)>(tr, ti, C, G);
        }
        fc_column<T, TJ, K, J + 1>(s, C, G);
    }
}

// dE/dr of one pair from its sums S = (F, Gz, Gx, Gy).  a = (z0 - i z) / r0 and
// b = (y - i x) / r0; the part of their derivatives along (a, b) itself is no
// rotation and drops out, which leaves dz0/dr e_k in a and the unit vectors.
__device__ __forceinline__ void fc_force(double (&o)[3], const double x, const double y, const double z,
                                         const double ar, const double ai, const double br, const double bi,
                                         const double (&S)[4], const SnapGeom &p)
{
    const double rsq = x * x + y * y + z * z, r = sqrt(rsq), rinv = 1.0 / r;
    const double r0inv = sqrt(ai * ai + br * br + bi * bi) * rinv;
    const double z0 = ar / r0inv;
    const double tscale = p.rfac0 * M_PI / (p.rcut - p.rmin0);
    const double dz = z0 * rinv - tscale * (rsq + z0 * z0) * rinv;
    double sfac = 1.0, dsfac = 0.0;
    if (p.switchflag == 1 && r > p.rmin0 && r <= p.rcut) {
        const double rf = M_PI / (p.rcut - p.rmin0);
        double sn, cs;
        sincos((r - p.rmin0) * rf, &sn, &cs);
        sfac = 0.5 * (cs + 1.0);
        dsfac = -0.5 * sn * rf;
    }
    const double c = 2.0 * sfac * p.wj * r0inv;
    const double rad = (2.0 * dsfac * p.wj * S[0] + c * dz * (ai * S[1] + br * S[2] - bi * S[3])) * rinv;
    o[0] = rad * x + c * (ai * S[2] - br * S[1] - ar * S[3]);
    o[1] = rad * y - c * (bi * S[1] + ar * S[2] + ai * S[3]);
    o[2] = rad * z + c * (ar * S[1] - bi * S[2] - br * S[3]);
}

// job K of the window's pairs on atoms a0 .. a0 + na - 1
template <typename T, int TJ, int K>
__device__ __forceinline__ void fc_job(const int a0, const int na, const typename cplx<T>::type *__restrict__ Y,
                                       const FcEntry *__restrict__ ent, typename cplx<T>::type *__restrict__ Cs,
                                       double4 *__restrict__ sums, const T *__restrict__ sab,
                                       const int *__restrict__ satom)
{
    if constexpr (K < FcJobs<TJ>::n) {
        constexpr UrJob jb = FcJobs<TJ>::at(K);
        constexpr int N = ur_count<TJ>(jb), B = fc_base<TJ>(K), NP = fc_pairs<T>(), NYH = yh_count(TJ);
        __syncthreads();   // the previous job's coefficients have been read
        for (int e = threadIdx.x; e < N * na; e += FC_THREADS) {
            const int k = e / na, sl = e - k * na, a = a0 + sl;
            const FcEntry &c = ent[B + k];
            fc_coeffs<T>(c, Y + (size_t)(a >> 5) * NYH * 32 + (a & 31) + c.k, Cs + 3 * k * fc_cap<T>() + sl);
        }
        __syncthreads();
#pragma unroll 1
        for (int q = threadIdx.x; q < NP; q += FC_THREADS) {
            const int atom = satom[q] - a0;
            if (atom < 0 || atom >= na) continue;
            UrState<T, TJ> s;
            s.ar = sab[q]; s.ai = sab[NP + q]; s.br = sab[2 * NP + q]; s.bi = sab[3 * NP + q];
            s.pr[0] = T(1);
            s.pi[0] = T(0);
            typename FAccSel<T>::type G[4];
#pragma unroll
            for (int k = 0; k < 4; k++) G[k].init(T(0));
            ur_chain<T, TJ, jb.mb, 0>(s);
            fc_column<T, TJ, K, (jb.mb == 0 ? 0 : 2 * jb.mb)>(s, Cs + atom, G);
            double4 v = K ? sums[q] : make_double4(0.0, 0.0, 0.0, 0.0);
            v.x += G[0].val();
            v.y += G[1].val();
            v.z += G[2].val();
            v.w += G[3].val();
            sums[q] = v;
        }
        fc_job<T, TJ, K + 1>(a0, na, Y, ent, Cs, sums, sab, satom);
    }
}

template <typename T, int TJ>
__global__ void __launch_bounds__(FC_THREADS, 2)
k_snap_fc(const double4 *__restrict__ prij, const double4 *__restrict__ pab, const int2 *__restrict__ pinfo,
          const int *__restrict__ pnum, SnapGeom gp, const typename cplx<T>::type *__restrict__ Y,
          double4 *__restrict__ dEslot)
{
    typedef typename cplx<T>::type T2;
    constexpr int NP = fc_pairs<T>(), CAP = fc_cap<T>();
    extern __shared__ __align__(16) unsigned char smraw[];
    double4 *sums = reinterpret_cast<double4 *>(smraw);                     // [pair]: F, Gz, Gx, Gy
    T2 *Cs = reinterpret_cast<T2 *>(sums + NP);                             // [entry][C0, Cx, Cy][slot]
    FcEntry *ent = reinterpret_cast<FcEntry *>(Cs + fc_most<TJ>() * 3 * CAP);
    T *sab = reinterpret_cast<T *>(ent + fc_base<TJ>(FcJobs<TJ>::n));       // [a, b][pair]
    int *satom = reinterpret_cast<int *>(sab + 4 * NP);                     // [pair]
    int *afirst = satom + NP;                                               // the window's first atom
    fc_entries<TJ, 0>(ent, threadIdx.x, FC_THREADS);
    const int npairs = *pnum;
    // windows of NP consecutive pairs (the loop bounds are uniform over the CTA)
    for (int base = blockIdx.x * NP; base < npairs; base += gridDim.x * NP) {
        if (threadIdx.x == 0) *afirst = INT_MAX;
        __syncthreads();
        for (int q = threadIdx.x; q < NP; q += FC_THREADS) {
            const int p = base + q;
            int atom = INT_MAX;
            if (p < npairs) {
                atom = pinfo[p].x;
                const double4 ab = pab[p];
                sab[q] = (T)ab.x;
                sab[NP + q] = (T)ab.y;
                sab[2 * NP + q] = (T)ab.z;
                sab[3 * NP + q] = (T)ab.w;
            }
            satom[q] = atom;
            const int first = __reduce_min_sync(0xffffffffu, atom);
            if ((threadIdx.x & 31) == 0) atomicMin(afirst, first);
        }
        __syncthreads();
        int a0 = *afirst;
        while (a0 != INT_MAX) {
            // the turn's last atom, and the first one of the next turn
            int last = a0, after = INT_MAX;
            for (int q = threadIdx.x & 31; q < NP; q += 32) {
                const int atom = satom[q];
                if (atom < a0 + CAP) last = max(last, atom);
                else after = min(after, atom);
            }
            const int na = __reduce_max_sync(0xffffffffu, last) - a0 + 1;
            after = __reduce_min_sync(0xffffffffu, after);
            fc_job<T, TJ, 0>(a0, na, Y, ent, Cs, sums, sab, satom);
            a0 = after;
        }
        // a thread's pairs are the ones it has summed
        for (int q = threadIdx.x; q < NP; q += FC_THREADS) {
            const int p = base + q;
            if (p >= npairs) continue;
            const double4 v = sums[q], r = prij[p], ab = pab[p];
            const double S[4] = {v.x, v.y, v.z, v.w};
            double o[3];
            fc_force(o, r.x, r.y, r.z, ab.x, ab.y, ab.z, ab.w, S, gp);
            dEslot[pinfo[p].y] = make_double4(o[0], o[1], o[2], 0.0);
        }
    }
}

}  // namespace mdp
