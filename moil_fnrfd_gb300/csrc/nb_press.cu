// nb_press.cu -- MOIL's pressure analysis terms (analysis/pressure.f, pressON) after an
// evaluation: per replica the diagonal of the molecular virial, split as pressure.f prints it,
//   virXX..ZZ    LJ pairs (pot/watwat_ewald.f:163-175, pot/cdie_ewald.f:441-453 and
//                555-566, image pairs symm/symwat_ewald.f:161-173, symm/symcdie_ewald.f:151-161)
//   V_PIdirXX..  real-space Ewald Coulomb pairs (watwat_ewald.f:196-204,
//                cdie_ewald.f:412-429, symwat_ewald.f:193-203)
//   V_PIrecXX..  reciprocal sum (pot/ewald_receip.f:799-807; k_press_zvir_f / _d in
//                nb_pme.cu)
//   V_PIrelXX..  PME force times the atom's position relative to its molecule's centre of
//                mass (ewald_receip.f:928-933)
// pressure.f:235-238 adds vir + dir + rec - rel; V_PIcor stays zero (its accumulation is
// commented out in cdie_ewald.f:165-170).
//
// Every pair term is F_ij,a (R_I - R_J)_a, R the centres of mass in the image the pair is
// taken in.  R_I - R_J is formed as r_ij - xrel_i + xrel_j from the pair's own minimum-image
// separation and the atoms' positions relative to their centres of mass (xrel), so no centre
// of mass is imaged.  Molecules are made whole by placing each atom at the minimum image of
// its displacement from the previous atom of its molecule (pressure.f joins them along bonds
// with checkANDmove, :985-1010), which needs consecutive atoms of a molecule closer than half
// the box.
//
// The pass reuses the evaluation's lists, site positions, PME records and PME gradient
// shares, with the pair predicates and the arithmetic of the energy kernels of the handle's
// precision.  On the mixed path the products with the centre-of-mass separations are FP32
// too, summed per lane in FP32 over at most NB_PCHUNK list entries, then as hi + lo pairs (an FP64
// operation per pair would cost more than the pair itself: the FP64 pipe is 1/64 of FP32); the
// plain path is FP64 throughout.  Water-water pairs are taken once, by their owner, with weight
// two; full lists hold every atom-atom pair twice; water-atom pairs are taken from the atom's
// side only with weight two; all are halved at the end.  The reciprocal part (spread, forward
// transforms, virial) runs on a second stream beside the pair kernels.  48 replicas (82,500
// waters), a call with its evaluation: 835 -> 675 us.
#include "nb_internal.h"
#include "nb_pair.cuh"

void nb_launch_pme_virial(NbCtx *c, cudaStream_t s, void *grid, double *v_col);

namespace {

#define NB_PCHUNK 32

// the pair arithmetic of each precision (as the energy kernels: MUFU rsqrt and the fitted
// erfc in FP32, libdevice in FP64)
template <typename T> struct PressMath;
template <> struct PressMath<float> {
    __device__ static float qq(const RepDev &R, int k) { return R.qq[k]; }
    __device__ static float w12(const RepDev &R) { return R.w12; }
    __device__ static float w6(const RepDev &R) { return R.w6; }
    __device__ static float c2a(const RepDev &R) { return R.c2a; }
    __device__ static float epstmp(const RepDev &R) { return (float)R.epstmp; }
    __device__ static float rsqrt(float x) { return nb_rsqrt_approx(x); }
    __device__ static float erfc_ex(const RepDev &R, float r2, float rinv, float *ex)
    {
        return nb_erfc_ex(R.alpha * r2 * rinv, r2 * R.ex2c, ex);
    }
};
template <> struct PressMath<double> {
    __device__ static double qq(const RepDev &R, int k) { return R.qqd[k]; }
    __device__ static double w12(const RepDev &R) { return R.w12d; }
    __device__ static double w6(const RepDev &R) { return R.w6d; }
    __device__ static double c2a(const RepDev &R) { return NB_TWO_OVER_SQRTPI * R.alphad; }
    __device__ static double epstmp(const RepDev &R) { return R.epstmp; }
    __device__ static double rsqrt(double x) { return ::rsqrt(x); }
    __device__ static double erfc_ex(const RepDev &R, double r2, double rinv, double *ex)
    {
        return nb_erfc_ex(R.alphad * r2 * rinv, 0.0, ex);
    }
};

// minus (dE_LJ/dr)/r of one pair with the LJ switch extension applied
template <typename T>
__device__ __forceinline__ T lj_mdf(const RepDev &R, T r2, T A, T B)
{
    const T s2 = (T)1 / r2, e1 = A - B;
    T df1 = (T)-6 * s2 * (A + e1);
    if (R.lj_switch && r2 > (T)R.ron2) {
        const T dd = (T)R.rv2 - r2;
        const T sw = dd * dd * ((T)R.rv2 + (T)2 * r2 - (T)3 * (T)R.ron2) * (T)R.swden;
        const T dsw = (T)12 * dd * ((T)R.ron2 - r2) * (T)R.swden;
        df1 = df1 * sw + e1 * dsw;
    }
    return -df1;
}

// positions relative to the centres of mass, in site order and the handle's precision (read beside
// the site positions); one thread per molecule, FP64 in xrel (caller order) until the centre is known
template <typename T>
__global__ void k_press_xrel(int nmol, const int *__restrict__ mol_off, const int *__restrict__ mol_atom,
                             const int *__restrict__ atom_rep, const RepDev *__restrict__ reps,
                             const double *__restrict__ coor, const double *__restrict__ mass,
                             const int *__restrict__ site_of, double *__restrict__ xrel, void *__restrict__ xsite_v)
{
    typedef typename vec4<T>::type T4;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nmol) return;
    const int b = mol_off[m], e = mol_off[m + 1];
    const RepDev &R = reps[atom_rep[mol_atom[b]]];
    double d[3] = {0.0, 0.0, 0.0}, sm[3] = {0.0, 0.0, 0.0}, M = 0.0;
    int prev = mol_atom[b];
    for (int k = b; k < e; ++k) {
        const int a = mol_atom[k];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            if (k > b) {
                const double t = coor[3 * (size_t)a + x] - coor[3 * (size_t)prev + x];
                d[x] += t - R.Ld[x] * rint(t * R.invLd[x]);
            }
            xrel[3 * (size_t)a + x] = d[x];
            sm[x] += mass[a] * d[x];
        }
        M += mass[a];
        prev = a;
    }
    const double im = M > 0.0 ? 1.0 / M : 0.0;
    const double com[3] = {sm[0] * im, sm[1] * im, sm[2] * im};
    for (int k = b; k < e; ++k) {
        const int a = mol_atom[k];
        const double *x = xrel + 3 * (size_t)a;
        T4 o;
        o.x = (T)(x[0] - com[0]); o.y = (T)(x[1] - com[1]); o.z = (T)(x[2] - com[2]); o.w = (T)0;
        ((T4 *)xsite_v)[site_of[a]] = o;
    }
}

// the six sums of a lane: FP32 as hi + lo pairs, FP64 plain
template <typename T> struct PressSum;
template <> struct PressSum<float> {
    float2 s[6] = {};
    __device__ void add(float f[6])
    {
#pragma unroll
        for (int k = 0; k < 6; ++k) { two_add(s[k], f[k]); f[k] = 0.f; }
    }
    template <int W> __device__ double total(int k)
    {
        const float2 a = sub_two_sum<W>(s[k]);
        return (double)a.x + (double)a.y;
    }
};
template <> struct PressSum<double> {
    double s[6] = {};
    __device__ void add(double f[6])
    {
#pragma unroll
        for (int k = 0; k < 6; ++k) { s[k] += f[k]; f[k] = 0.0; }
    }
    template <int W> __device__ double total(int k) { return sub_sum<W>(s[k]); }
};

// Coulomb force over the nine site pairs of two waters, d the O-O vector, j1 and j2 the partner's H
// offsets: FP32 with eight of the nine packed two by two, as in the energy kernels
template <typename T> struct PressK;
template <> struct PressK<float> {
    WaterK K;
    float qOO, qOH, qHH;
    __device__ PressK(const RepDev &R)
        : K{held(ERFCX_P * R.alpha), held(R.ex2c), held(R.c2a)}, qOO(held(R.qq[0])), qOH(held(R.qq[1])), qHH(held(R.qq[2]))
    {
    }
};
template <> struct PressK<double> {
    const RepDev &R;
    __device__ PressK(const RepDev &R_) : R(R_) {}
};
__device__ __forceinline__ void water_coulomb(const PressK<float> &P, const float hi[2][3], const float d[3], float4 j1,
                                              float4 j2, float fc[3])
{
    const WaterK &K = P.K;
    const float qOO = P.qOO, qOH = P.qOH, qHH = P.qHH;
    const float rr2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    float e;
    const float m0 = ewald1(K, rr2, nb_rsqrt_approx(rr2), qOO, e);
    float2 F[3] = {f2(m0 * d[0], 0.f), f2(m0 * d[1], 0.f), f2(m0 * d[2], 0.f)}, ee;
    const float q1[3] = {d[0] - j1.x, d[1] - j1.y, d[2] - j1.z}, q2[3] = {d[0] - j2.x, d[1] - j2.y, d[2] - j2.z};
    auto two = [&](float2 x, float2 y, float2 z, float qq) {
        const float2 m = ewald2(K, __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z))), f2(qq), ee);
        F[0] = __ffma2_rn(m, x, F[0]); F[1] = __ffma2_rn(m, y, F[1]); F[2] = __ffma2_rn(m, z, F[2]);
    };
    two(f2(q1[0], q2[0]), f2(q1[1], q2[1]), f2(q1[2], q2[2]), qOH);
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const float *q = s == 0 ? d : (s == 1 ? q1 : q2);
        two(f2(hi[0][0] + q[0], hi[1][0] + q[0]), f2(hi[0][1] + q[1], hi[1][1] + q[1]),
            f2(hi[0][2] + q[2], hi[1][2] + q[2]), s == 0 ? qOH : qHH);
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) fc[x] = F[x].x + F[x].y;
}
__device__ __forceinline__ void water_coulomb(const PressK<double> &P, const double hi[2][3], const double d[3],
                                              double4 j1, double4 j2, double fc[3])
{
    const RepDev &R = P.R;
    typedef PressMath<double> M;
    const double hj[3][3] = {{0, 0, 0}, {j1.x, j1.y, j1.z}, {j2.x, j2.y, j2.z}};
    const double c2a = M::c2a(R);
#pragma unroll
    for (int x = 0; x < 3; ++x) fc[x] = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            double v[3];
#pragma unroll
            for (int x = 0; x < 3; ++x) v[x] = (a ? hi[a ? a - 1 : 0][x] : 0.0) + d[x] - hj[b][x];
            const double rr2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2], rinv = M::rsqrt(rr2);
            double ex;
            const double erfcv = M::erfc_ex(R, rr2, rinv, &ex);
            const double qq = M::qq(R, (a == 0 && b == 0) ? 0 : ((a == 0 || b == 0) ? 1 : 2));
            const double mdf = (qq * erfcv * rinv + qq * c2a * ex) * rinv * rinv;   // minus dE/dr / r
#pragma unroll
            for (int x = 0; x < 3; ++x) fc[x] += mdf * v[x];
        }
}

// Water-water pairs (watwat_ewald.f semantics, water charges of RepDev): 9 Coulomb site pairs and the
// O-O LJ pair of every molecule inside the O-O cutoff, each pair once, by its owner (the terms are
// the same from both sides).  Eight lanes share a water's row: owned in-cutoff entries are
// compacted into shared memory with their image-shifted O-O vectors, then the lanes take one
// entry each, so no lane waits through pairs that others skip.  Bound: FP32 issue.  One water per
// thread over full rows took 239 us for 82,500 waters, this 141 (the FP64 path the same way).
#define PW_BLOCK 128
#define PW_LANES 8
#define PW_CAP 64
template <typename T, typename E>
__global__ void __launch_bounds__(PW_BLOCK, 4) k_press_water(int nW, const RepDev *__restrict__ reps,
                                                             const int *__restrict__ site_rep, const void *pos_v,
                                                             const void *woff_v, const int2 *__restrict__ wl1_cnt,
                                                             const void *__restrict__ wl1, int cap_row,
                                                             const void *xsite_v, double *__restrict__ pu)
{
    typedef typename vec4<T>::type T4;
    typedef PressMath<T> M;
    __shared__ T4 sD[PW_BLOCK / PW_LANES][PW_CAP];
    __shared__ int sJ[PW_BLOCK / PW_LANES][PW_CAP];
    const int lane = threadIdx.x & 31, sub = threadIdx.x & (PW_LANES - 1), w = threadIdx.x / PW_LANES;
    const int iw = blockIdx.x * (PW_BLOCK / PW_LANES) + w;
    const bool act = iw < nW;
    const int i = act ? iw : nW - 1;         // idle lanes of the last block: an empty row, no output
    const T4 *pos = (const T4 *)pos_v, *woff = (const T4 *)woff_v, *xsite = (const T4 *)xsite_v;
    const RepDev &R = reps[site_rep[3 * i]];
    const T4 oi = pos[3 * i], h1 = woff[3 * i + 1], h2 = woff[3 * i + 2], xi = xsite[3 * i];
    const T hi[2][3] = {{h1.x, h1.y, h1.z}, {h2.x, h2.y, h2.z}};
    const T rmax2 = (T)R.rmax2, rv2 = (T)R.rv2;
    const PressK<T> P(R);
    PressSum<T> v;
    T f[6] = {(T)0, (T)0, (T)0, (T)0, (T)0, (T)0};
    auto work_off = [&](int cnt) {
        __syncwarp();
        for (int e = sub; e < cnt; e += PW_LANES) {
            const T4 D = sD[w][e];
            const int j = sJ[w][e];
            const T4 xj = xsite[3 * (size_t)j];
            const T d[3] = {D.x, D.y, D.z}, rm[3] = {d[0] - xi.x + xj.x, d[1] - xi.y + xj.y, d[2] - xi.z + xj.z};
            T fc[3];
            water_coulomb(P, hi, d, woff[3 * (size_t)j + 1], woff[3 * (size_t)j + 2], fc);
#pragma unroll
            for (int x = 0; x < 3; ++x) f[3 + x] += fc[x] * rm[x];
            if (D.w <= rv2) {
                const T s2 = (T)1 / D.w, s6 = s2 * s2 * s2;
                const T m1 = lj_mdf<T>(R, D.w, M::w12(R) * s6 * s6, M::w6(R) * s6);
#pragma unroll
                for (int x = 0; x < 3; ++x) f[x] += m1 * d[x] * rm[x];
            }
        }
        v.add(f);
        __syncwarp();
    };
    const W1Row<E> row(wl1_cnt, wl1, cap_row, i, R.wat0);
    const int n = act ? row.n : 0, il = i - R.wat0;
    int cnt = 0, jn = sub < n ? row.at(sub) : -1;
    for (int k = sub; __any_sync(0xffffffffu, k - sub < n); k += PW_LANES) {
        const int j = jn;
        jn = k + PW_LANES < n ? row.at(k + PW_LANES) : -1;     // the next entry on its way
        bool in = false;
        T4 D;
        if (j >= 0 && nb_half_owner(il, j - R.wat0) == il) {
            const T4 oj = pos[3 * (size_t)j];
            T d[3] = {oi.x - oj.x, oi.y - oj.y, oi.z - oj.z};
#pragma unroll
            for (int x = 0; x < 3; ++x) d[x] = nb_shift(R, x, d[x], nb_rint(d[x] * rep_invL<T>(R, x)));
            D.x = d[0]; D.y = d[1]; D.z = d[2];
            D.w = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
            in = D.w <= rmax2;
        }
        const unsigned m = (__ballot_sync(0xffffffffu, in) >> (lane - sub)) & ((1u << PW_LANES) - 1u);
        if (in) {
            const int p = cnt + __popc(m & ((1u << sub) - 1u));
            sD[w][p] = D;
            sJ[w][p] = j;
        }
        cnt += __popc(m);
        if (__any_sync(0xffffffffu, cnt > PW_CAP - PW_LANES)) { work_off(cnt); cnt = 0; }
    }
    work_off(cnt);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const double s = v.template total<PW_LANES>(k);
        if (act && sub == k) pu[6 * (size_t)i + k] = 2.0 * s;
    }
}

// non-water atom per warp, lanes over its X list (non-water atoms and water sites), the pair
// predicate of the energy kernels' atom_pair (cdie_ewald.f list1/2/3, nbond.f:115-126)
template <typename T>
__global__ void k_press_atom(int nA, int nW, const RepDev *__restrict__ reps, const int *__restrict__ site_rep,
                             const void *pos_v, const void *lj_v, const unsigned *__restrict__ sflags,
                             const int *__restrict__ xl_off, const int *__restrict__ xl, int capx, const void *xsite_v,
                             double *__restrict__ pu)
{
    typedef typename vec4<T>::type T4;
    typedef typename cplx<T>::type T2;
    typedef PressMath<T> M;
    const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= nA) return;
    const T4 *pos = (const T4 *)pos_v, *xsite = (const T4 *)xsite_v;
    const T2 *lj = (const T2 *)lj_v;
    const int si = 3 * nW + k;
    const RepDev &R = reps[site_rep[si]];
    const T4 xi = pos[si];
    const T2 lji = lj[si];
    const unsigned fi = sflags[si];
    const T4 xa = xsite[si];
    const T rv2 = (T)R.rv2, re2 = (T)R.re2, rmax2 = (T)R.rmax2, c2a = M::c2a(R);
    PressSum<T> v;
    T f[6] = {(T)0, (T)0, (T)0, (T)0, (T)0, (T)0};
    int cnt = 0;
    for (int q = min(xl_off[k], capx) + lane; q < min(xl_off[k + 1], capx); q += 32) {
        const int s = xl[q];
        const T4 xj = pos[s];
        T d[3] = {xi.x - xj.x, xi.y - xj.y, xi.z - xj.z};
#pragma unroll
        for (int x = 0; x < 3; ++x) d[x] = nb_shift(R, x, d[x], nb_rint(d[x] * rep_invL<T>(R, x)));
        const T r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const unsigned fj = sflags[s];
        const bool hr = !R.arith && R.hvdw0 && ((fi | fj) & SF_HTINY) && r2 < re2;
        const bool do_lj = r2 < rv2 && !hr;
        T qq = xi.w * xj.w;
        const bool do_el = r2 < rmax2 && qq != (T)0;
        if (!do_lj && !do_el) continue;
        const T rinv = M::rsqrt(r2), s2 = rinv * rinv;
        T m_el = (T)0, m_lj = (T)0;   // minus (dE/dr)/r of each part
        if (do_el) {
            T exv;
            const T erfcv = M::erfc_ex(R, r2, rinv, &exv);
            qq *= M::epstmp(R);
            m_el = (qq * erfcv * rinv + qq * c2a * exv) * s2;
        }
        if (do_lj) {
            const T2 ljj = lj[s];
            const T s6 = s2 * s2 * s2;
            T A, B;
            if (!R.arith) {
                A = lji.x * ljj.x * s6 * s6;
                B = lji.y * ljj.y * s6;
            } else {
                const T aa = lji.x * ljj.x, sg = (T)0.5 * (lji.y + ljj.y);
                T b1 = sg * sg * sg;
                b1 = b1 * b1;
                B = aa * b1 * s6;
                A = aa * b1 * b1 * s6 * s6;
            }
            m_lj = lj_mdf<T>(R, r2, A, B);
        }
        const T w = s < 3 * nW ? (T)2 : (T)1;   // water partners: this side only
        const T4 xb = xsite[s];
        const T rm[3] = {d[0] - xa.x + xb.x, d[1] - xa.y + xb.y, d[2] - xa.z + xb.z};
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            f[x] += w * m_lj * d[x] * rm[x];
            f[3 + x] += w * m_el * d[x] * rm[x];
        }
        if (++cnt == NB_PCHUNK) { v.add(f); cnt = 0; }
    }
    __syncwarp();     // lists' remainders: the lanes together again
    v.add(f);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const double s = v.template total<32>(m);
        if (lane == m) pu[6 * (size_t)(nW + k) + m] = s;
    }
}

// V_PIrel of a site: the PME force (minus the gradient share the evaluation adds) times xrel
template <typename T>
__device__ __forceinline__ void press_rel(int s, int a, const RepDev &R, const void *part_v, const double *q,
                                          const void *xsite_v, double acc[3])
{
    const typename vec4<T>::type x = ((const typename vec4<T>::type *)xsite_v)[s];
    if constexpr (sizeof(T) == 4) {
        // one float4 per site from k_pme_gather_f, scaled by q fc n_d / L_d
        const float4 p = ((const float4 *)part_v)[s];
        const float qs = -(float)q[a];
        acc[0] += (double)(qs * R.pme_gs[0] * p.x * x.x);
        acc[1] += (double)(qs * R.pme_gs[1] * p.y * x.y);
        acc[2] += (double)(qs * R.pme_gs[2] * p.z * x.z);
    } else {
        // four plane slots of three per site from k_plane_inv
        const double *p = (const double *)part_v + 12 * (size_t)s;
        const double qf = q[a] * R.fcd;
        const double sc[3] = {qf * R.n1 * R.invLd[0], qf * R.n2 * R.invLd[1], qf * R.n3 * R.invLd[2]};
        const double xr[3] = {x.x, x.y, x.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) acc[d] += -sc[d] * (p[d] + p[3 + d] + p[6 + d] + p[9 + d]) * xr[d];
    }
}

// Sums per replica in a fixed order: press_blocks blocks per replica (by its own size, whatever else
// the handle holds), each strided slots per thread and a halving tree, then k_press_final over the
// blocks.  One block per replica of up to 4,000 waters took 38 us (and the V_PIrel terms a pass of
// their own, 6); this 19 and 4.
#define NB_PR_THREADS 256
__host__ __device__ __forceinline__ int press_blocks(const RepDev &R)
{
    const int b = (3 * R.nwat + R.noth + 1023) / 1024;
    return b < 1 ? 1 : (b > 64 ? 64 : b);
}
template <typename T>
__global__ void __launch_bounds__(NB_PR_THREADS) k_press_reduce(int nW, const RepDev *__restrict__ reps,
                                                               const int *__restrict__ site_orig,
                                                               const void *part_v, const double *__restrict__ q,
                                                               const void *xsite_v, const double *__restrict__ pu,
                                                               const double *__restrict__ v_col,
                                                               const int *__restrict__ col_begin,
                                                               double *__restrict__ out)
{
    __shared__ double red[12][NB_PR_THREADS];
    const int r = blockIdx.x, t = threadIdx.x;     // (replicas along x: the other axes end at 65,535)
    const RepDev &R = reps[r];
    if ((int)blockIdx.y >= press_blocks(R)) return;
    const int first = blockIdx.y * NB_PR_THREADS + t, stride = press_blocks(R) * NB_PR_THREADS;
    double acc[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) acc[k] = 0.0;
    const int u0[2] = {R.wat0, nW + R.oth0}, nu[2] = {R.nwat, R.noth};
    const int s0[2] = {3 * R.wat0, 3 * nW + R.oth0}, ns[2] = {3 * R.nwat, R.noth};
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        for (int u = first; u < nu[p]; u += stride) {
            const double *v = pu + 6 * (size_t)(u0[p] + u);
#pragma unroll
            for (int k = 0; k < 6; ++k) acc[k] += v[k];
        }
        for (int u = first; u < ns[p]; u += stride)
            press_rel<T>(s0[p] + u, site_orig[s0[p] + u], R, part_v, q, xsite_v, acc + 9);
    }
    for (int w = col_begin[r] + first; w < col_begin[r + 1]; w += stride) {
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[6 + k] += v_col[3 * (size_t)w + k];
    }
#pragma unroll
    for (int k = 0; k < 12; ++k) red[k][t] = acc[k];
    __syncthreads();
    for (int h = NB_PR_THREADS / 2; h > 0; h >>= 1) {
        if (t < h)
#pragma unroll
            for (int k = 0; k < 12; ++k) red[k][t] += red[k][t + h];
        __syncthreads();
    }
    if (t < 12) out[12 * ((size_t)r * gridDim.y + blockIdx.y) + t] = red[t][0];
}

__global__ void k_press_final(int n, int nsplit, const RepDev *__restrict__ reps, const double *__restrict__ part,
                              double *__restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n) return;
    const int r = x / 12, k = x - 12 * r;
    double s = 0.0;
    for (int b = 0; b < press_blocks(reps[r]); ++b) s += part[12 * ((size_t)r * nsplit + b) + k];
    out[x] = (k < 9 ? 0.5 : 1.0) * s;
}

template <typename T>
void pressure_t(NbCtx *c, const double *d_coor, double *d_out)
{
    cudaStream_t s = c->stream, pme = c->stream2;
    const int B = 128;
    // the reciprocal part beside the pair kernels
    cudaEventRecord(c->ev_fork, s);
    cudaStreamWaitEvent(pme, c->ev_fork, 0);
    nb_launch_pme_virial(c, pme, c->d_press_grid, c->d_press_col);
    cudaEventRecord(c->ev_join, pme);
    if (c->nmol > 0)
        k_press_xrel<T><<<(c->nmol + 31) / 32, 32, 0, s>>>(c->nmol, c->d_mol_off, c->d_mol_atom, c->d_atom_rep, c->d_reps,
                                                           d_coor, c->d_mass, c->d_site_of, c->d_xrel, c->d_xsite);
    if (c->nW > 0) {
        const int wpb = PW_BLOCK / PW_LANES;
        (c->row16 ? k_press_water<T, unsigned short> : k_press_water<T, int>)<<<(int)((c->nW + wpb - 1) / wpb), PW_BLOCK, 0,
                                                                              s>>>(
            (int)c->nW, c->d_reps, c->d_site_rep, c->d_pos, c->d_woff, c->d_wl1_cnt, c->d_wl1, c->cap_row1,
            c->d_xsite, c->d_press_unit);
    }
    if (c->nA > 0)
        k_press_atom<T><<<(int)((c->nA + B / 32 - 1) / (B / 32)), B, 0, s>>>(
            (int)c->nA, (int)c->nW, c->d_reps, c->d_site_rep, c->d_pos, c->d_site_lj, c->d_site_flags, c->d_xl_off,
            c->d_xl, cap_int(c->cap_xl), c->d_xsite, c->d_press_unit);
    cudaStreamWaitEvent(s, c->ev_join, 0);
    k_press_reduce<T><<<dim3(c->nrep, c->press_split), NB_PR_THREADS, 0, s>>>(
        (int)c->nW, c->d_reps, c->d_site_orig, c->d_part, c->d_q, c->d_xsite, c->d_press_unit, c->d_press_col,
        c->d_col_begin, c->d_press_part);
    k_press_final<<<(12 * c->nrep + B - 1) / B, B, 0, s>>>(12 * c->nrep, c->press_split, c->d_reps, c->d_press_part, d_out);
}

}  // namespace

int nb_press_split(const NbCtx *c)
{
    int most = 1;
    for (int r = 0; r < c->nrep; ++r) most = std::max(most, press_blocks(c->rd[r]));
    return most;
}

int nb_pressure(NbCtx *c, const double *d_coor, double *d_out)
{
    if (c->precision == MOIL_NB_FP64) pressure_t<double>(c, d_coor, d_out);
    else pressure_t<float>(c, d_coor, d_out);
    NB_CUDA_OK(c, cudaGetLastError());
    return MOIL_NB_OK;
}
