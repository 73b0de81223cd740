// nb_realspace.cu -- real-space LJ + erfc-Coulomb, exclusion/1-4 corrections, finalize.
//
// Pair semantics are MOIL's predicate evaluated at the current coordinates:
//   water-water   pot/watwat_ewald.f:131-612 (+ images, symm/symwat_ewald.f): the molecule
//                 pair is in iff O-O r^2 <= max(cutvdw2, cutele2); then all 9 site pairs get
//                 erfc-Coulomb with the O-O image shift and no per-site cutoff, O-O LJ if
//                 r^2 <= cutvdw2.
//   other pairs   pot/cdie_ewald.f:313-671 (+ symm/symcdie_ewald.f) with the lists of
//                 pot/nbond.f:115-149: LJ iff r^2 < cutvdw2 (and not the geometric hydrogen
//                 rule inside cutele2), Coulomb iff both charged and r^2 < max(cutvdw2, cutele2).
//   primary vs image: a pair whose minimum-image shift is zero is a primary-box pair
//                 (e_vdw/e_el); any other shift is one of MOIL's translated images
//                 (e_vsym/e_lsym).
// Lists are full (each pair appears under both atoms); a water or atom owns its own gradient,
// so nothing is written twice and no atomics are needed, except where a kernel evaluates each
// water pair once (k_water_h, k_water_d).  Energies are halved at the end.
#include "nb_internal.h"
#include "nb_grad.cuh"
#include "nb_pair.cuh"

namespace {

#define CHUNK 64

// FP64 path: one non-water-type pair (cdie_ewald list1/2/3 semantics); d already minimum-imaged
// vir receives MOIL's LJ virial term of the pair, -df1 r^2 (cdie_ewald_press.f:413-419)
__device__ __forceinline__ double atom_pair(const RepDev &R, double r2, double qi, double qj, double e12i, double e6i,
                                            double e12j, double e6j, unsigned fi, unsigned fj, double &eel, double &elj,
                                            double &vir, int &npair)
{
    bool hr = !R.arith && R.hvdw0 && ((fi | fj) & SF_HTINY) && r2 < (double)R.re2;
    bool lj = r2 < (double)R.rv2 && !hr;
    double qq = qi * qj;
    bool el = r2 < (double)R.rmax2 && qq != 0.0;
    if (!lj && !el) return 0.0;
    ++npair;
    double rinv = nb_rsqrt(r2);
    double s2 = rinv * rinv;
    double df = 0;
    if (el) {
        double x = R.alphad * r2 * rinv;
        double ex;
        double erfcv = nb_erfc_ex(x, r2 * (double)R.ex2c, &ex);
        qq *= R.epstmp;
        double e = qq * erfcv * rinv;
        df = -(e + qq * (double)R.c2a * ex) * s2;
        eel += e;
    }
    if (lj) {
        double s6 = s2 * s2 * s2, A, B;
        if (!R.arith) {
            A = e12i * e12j * s6 * s6;
            B = e6i * e6j * s6;
        } else {
            double aa = e12i * e12j, sg = 0.5 * (e6i + e6j);
            double b1 = sg * sg * sg;
            b1 = b1 * b1;
            B = aa * b1 * s6;
            A = aa * b1 * b1 * s6 * s6;
        }
        double e1 = A - B;
        double df1 = -6.0 * s2 * (A + e1);
        lj_switch_apply<double>(R, r2, e1, df1);
        elj += e1;
        vir -= df1 * r2;
        df += df1;
    }
    return df;
}

__device__ __forceinline__ void min_image(const RepDev &R, double &dx, double &dy, double &dz, bool &img)
{
    const double nx = nb_rint(dx * R.invLd[0]), ny = nb_rint(dy * R.invLd[1]), nz = nb_rint(dz * R.invLd[2]);
    dx = nb_shift(R, 0, dx, nx);
    dy = nb_shift(R, 1, dy, ny);
    dz = nb_shift(R, 2, dz, nz);
    img = (nx != 0.0) | (ny != 0.0) | (nz != 0.0);
}

__device__ __forceinline__ void flush(float g[], long long G[], int n)
{
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        if (k < n) { G[k] += nb_fix(g[k]); g[k] = 0.f; }
    }
}
// water sites of molecule i against its W2 list of non-water atoms (entries first, first +
// stride, ...): atom semantics per site pair; partial gradients and energies go to g / e4, which
// already hold cnt entries, flushed every CHUNK entries and left to the caller after the last
template <typename Flush>
__device__ __forceinline__ void water_vs_atoms(const RepDev &R, int i, const double4 *pos,
                                               const void *lj_v, const unsigned *__restrict__ sflags,
                                               const int *__restrict__ wl2_off, const int *__restrict__ wl2, int cap2,
                                               int first, int stride, int cnt, double g[9], double e4[4], int &npair,
                                               Flush &flush_all)
{
    // an overflowed list (offsets past the capacity) is read within the buffer; the
    // evaluation reports the overflow and is redone with a larger one
    const int q0 = min(wl2_off[i], cap2), q1 = min(wl2_off[i + 1], cap2);
    if (q0 >= q1) return;
    const double2 *lj = (const double2 *)lj_v;
    const double4 si[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    const double2 lji[3] = {lj[3 * i], lj[3 * i + 1], lj[3 * i + 2]};
    const unsigned fi[3] = {sflags[3 * i], sflags[3 * i + 1], sflags[3 * i + 2]};
    for (int k = q0 + first; k < q1; k += stride) {
        nb_prefetch_l1(wl2 + min(k + 32, q1 - 1));
        int s = wl2[k];
        double4 xj = pos[s];
        double2 ljj = lj[s];
        unsigned fj = sflags[s];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            double dx = si[a].x - xj.x, dy = si[a].y - xj.y, dz = si[a].z - xj.z;
            bool img;
            min_image(R, dx, dy, dz, img);
            double r2 = dx * dx + dy * dy + dz * dz;
            double eel = 0, elj = 0, vir = 0;   // the virial of these pairs is counted by k_atom_d
            double df = atom_pair(R, r2, si[a].w, xj.w, lji[a].x, lji[a].y, ljj.x, ljj.y, fi[a], fj, eel, elj, vir,
                                npair);
            g[3 * a] += df * dx;
            g[3 * a + 1] += df * dy;
            g[3 * a + 2] += df * dz;
            e4[img ? 1 : 0] += elj;
            e4[img ? 3 : 2] += eel;
        }
        if (++cnt == CHUNK) { flush_all(); cnt = 0; }
    }
}

// FP32: the H sites packed two by two on the FP32x2 pipe, their LJ part skipped for waters whose
// hydrogens carry none.  Water stage of 8 systems of 7,020 waters and 2,496 atoms: three scalar pairs
// per entry 208 us, this 182, with records one entry ahead 170.
template <typename Flush>
__device__ __forceinline__ void water_vs_atoms(const RepDev &R, const AtomK &A, int i, const float4 *pos, const void *lj_v,
                                               const unsigned *__restrict__ sflags, const int *__restrict__ wl2_off,
                                               const int *__restrict__ wl2, int cap2, int first, int stride, int &cnt,
                                               float g[9], float e4[4], int &npair, Flush &flush_all)
{
    const int q0 = min(wl2_off[i], cap2), q1 = min(wl2_off[i + 1], cap2);
    if (q0 >= q1) return;
    const float2 *lj = (const float2 *)lj_v;
    const float4 o = pos[3 * i], h1 = pos[3 * i + 1], h2 = pos[3 * i + 2];
    const float2 ljo = lj[3 * i], lj1 = lj[3 * i + 1], lj2 = lj[3 * i + 2];
    const float qo = o.w * A.ke;
    const float2 qh = f2(h1.w * A.ke, h2.w * A.ke);
    const unsigned to = A.tiny ? sflags[3 * i] & SF_HTINY : 0, t1 = A.tiny ? sflags[3 * i + 1] & SF_HTINY : 0,
                   t2 = A.tiny ? sflags[3 * i + 2] & SF_HTINY : 0;
    const bool hlj = lj1.x != 0.f || lj2.x != 0.f || (!A.arith && (lj1.y != 0.f || lj2.y != 0.f));
    if (q0 + first >= q1) return;
    // the next entry's record is on its way while one is worked on, its index one further ahead
    auto entry = [&](int k) { return wl2[min(k, q1 - 1)]; };
    int sb = entry(q0 + first), sn = entry(q0 + first + stride);
    float4 xb = pos[sb];
    float2 lb = lj[sb];
    for (int k = q0 + first; k < q1; k += stride) {
        const int s = sb;
        const float4 xj = xb;
        const float2 ljj = lb;
        sb = sn;
        xb = pos[sb]; lb = lj[sb];
        sn = entry(k + 2 * stride);
        const unsigned fj = A.tiny ? sflags[s] & SF_HTINY : 0;
        float eel, elj, vir;      // the virial of these pairs is counted by k_atom_f
        bool img;
        {
            float dx = o.x - xj.x, dy = o.y - xj.y, dz = o.z - xj.z;
            A.image(dx, dy, dz, img);
            const float m = A.pair(R, dx * dx + dy * dy + dz * dz, qo * xj.w, ljo, ljj, (to | fj) != 0, eel, elj, vir, npair);
            g[0] = fmaf(-m, dx, g[0]); g[1] = fmaf(-m, dy, g[1]); g[2] = fmaf(-m, dz, g[2]);
            e4[0] += img ? 0.f : elj; e4[1] += img ? elj : 0.f;
            e4[2] += img ? 0.f : eel; e4[3] += img ? eel : 0.f;
        }
        float2 x = f2(h1.x - xj.x, h2.x - xj.x), y = f2(h1.y - xj.y, h2.y - xj.y), z = f2(h1.z - xj.z, h2.z - xj.z);
        float2 nx, ny, nz;
        A.image2(x, y, z, nx, ny, nz);
        const float2 r2 = __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z)));
        const float2 qq = __fmul2_rn(qh, f2(xj.w));
        const bool el1 = r2.x < A.rmax2 && qq.x != 0.f, el2 = r2.y < A.rmax2 && qq.y != 0.f;
        const bool v1 = r2.x < A.rv2 && !((t1 | fj) && r2.x < A.re2), v2 = r2.y < A.rv2 && !((t2 | fj) && r2.y < A.re2);
        npair += (int)(el1 || v1) + (int)(el2 || v2);
        if (el1 || el2 || (hlj && (v1 || v2))) {
            float2 e, m = ewald2(A.K, r2, qq, e);
            m = f2(el1 ? m.x : 0.f, el2 ? m.y : 0.f);
            e = f2(el1 ? e.x : 0.f, el2 ? e.y : 0.f);
            const bool i1 = (nx.x != 0.f) | (ny.x != 0.f) | (nz.x != 0.f), i2 = (nx.y != 0.f) | (ny.y != 0.f) | (nz.y != 0.f);
            if (hlj) {
                float l1 = 0.f, l2 = 0.f;
                if (v1) m.x += A.lj(R, r2.x, nb_rsqrt_approx(r2.x), lj1, ljj, l1);
                if (v2) m.y += A.lj(R, r2.y, nb_rsqrt_approx(r2.y), lj2, ljj, l2);
                e4[0] += (i1 ? 0.f : l1) + (i2 ? 0.f : l2);
                e4[1] += (i1 ? l1 : 0.f) + (i2 ? l2 : 0.f);
            }
            e4[2] += (i1 ? 0.f : e.x) + (i2 ? 0.f : e.y);
            e4[3] += (i1 ? e.x : 0.f) + (i2 ? e.y : 0.f);
            g[3] = fmaf(-m.x, x.x, g[3]); g[4] = fmaf(-m.x, y.x, g[4]); g[5] = fmaf(-m.x, z.x, g[5]);
            g[6] = fmaf(-m.y, x.y, g[6]); g[7] = fmaf(-m.y, y.y, g[7]); g[8] = fmaf(-m.y, z.y, g[8]);
        }
        if (++cnt == CHUNK) { flush_all(); cnt = 0; }
    }
}

// ---------------------------------------------------------------------------------
// Water kernels: W1 (water-water, 9 site pairs) then W2 (water sites x other atoms).  FP32 partial gradients
// and energies are flushed every CHUNK list entries of a lane, gradients as int64 fixed point, energies
// as hi + lo pairs.
#define WBLOCK 128

// Plain FP64 path: one warp per water.  Bound: the FP64 pipe (two lanes per clock and SM), about
// 120 FP64 instructions per site pair, so every molecule pair is evaluated once, by its owner
// (nb_half_owner on the full rows), and a warp's 32 lanes share one water's pairs: the owned
// in-cutoff entries are compacted into shared memory (their image-shifted O-O vectors with
// them), and the lanes take (partner site, entry) items, three site pairs each, so about 50
// entries fill five rounds of 32 items.  Gradients of both sides go to int64 arrays (cleared before the
// launch) with atomics: integer sums, independent of their order, of parts rounded to 2^-43 (nb_fine:
// 32 lanes and about 65 partner shares per site; at 2^-33 each the sums were off by up to 2.5e-9).
// erfc(x) is exp(-x^2) erfcx(x), one exponential for the energy and the force.  A whole evaluation: 216
// waters 3258 -> 226 us, 1,334 waters 3867 -> 485 us (before: one water per thread, full lists).
#define WARPS64 2
#define WBUF64 96
template <typename E>
__global__ void __launch_bounds__(32 * WARPS64) k_water_d(int nW, const RepDev *__restrict__ reps,
                                                          const int *__restrict__ site_rep,
                                                          const double4 *__restrict__ pos,
                                                          const double4 *__restrict__ woff, const void *lj_v,
                                                          const unsigned *__restrict__ sflags,
                                                          const int2 *__restrict__ wl1_cnt,
                                                          const void *__restrict__ wl1, int cap_row,
                                                          const int *__restrict__ wl2_off,
                                                          const int *__restrict__ wl2, int cap2,
                                                          unsigned long long *__restrict__ grad,
                                                          unsigned long long *__restrict__ fine,
                                                          double *__restrict__ e_unit)
{
    __shared__ double sD[WARPS64][3][WBUF64];
    __shared__ int sJ[WARPS64][WBUF64];      // partner, negative (~partner) for an image pair
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * WARPS64 + warp;
    if (i >= nW) return;
    double (*D)[WBUF64] = sD[warp];
    int *J = sJ[warp];
    const RepDev &R = reps[site_rep[3 * i]];
    const double4 oi0 = pos[3 * i], oi1 = woff[3 * i + 1], oi2 = woff[3 * i + 2];
    const double hi[2][3] = {{oi1.x, oi1.y, oi1.z}, {oi2.x, oi2.y, oi2.z}};
    double g[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) g[k] = 0.0;
    double e4[6] = {0, 0, 0, 0, 0, 0};   // LJ prim, LJ img, Coulomb prim, Coulomb img, LJ virial prim, img
    int npair = 0;
    const double rmax2 = (double)R.rmax2, rv2 = (double)R.rv2, alpha = R.alphad, c2a = (double)R.c2a;
    const double qOO = R.qqd[0], qOH = R.qqd[1], qHH = R.qqd[2], w12 = R.w12d, w6 = R.w6d;
    const W1Row<E> L1(wl1_cnt, wl1, cap_row, i, R.wat0);
    // the buffered entries: items b-major, so a round's lanes share a partner site (almost)
    auto work_off = [&](int cnt) {
        __syncwarp();
        for (int it = lane; it < 3 * cnt; it += 32) {
            const int b = it >= 2 * cnt ? 2 : (it >= cnt ? 1 : 0), e = it - b * cnt;
            const int jj = J[e];
            const bool img = jj < 0;
            const int j = img ? ~jj : jj;
            double q[3] = {D[0][e], D[1][e], D[2][e]};
            if (b) {
                const double4 oj = woff[3 * (size_t)j + b];
                q[0] -= oj.x; q[1] -= oj.y; q[2] -= oj.z;
            }
            double H[3] = {0.0, 0.0, 0.0}, e_el = 0.0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const double dx = a ? hi[a - 1][0] + q[0] : q[0], dy = a ? hi[a - 1][1] + q[1] : q[1],
                             dz = a ? hi[a - 1][2] + q[2] : q[2];
                const double rr2 = dx * dx + dy * dy + dz * dz, rinv = rsqrt(rr2), s2 = rinv * rinv;
                const double x = alpha * rr2 * rinv, ex = exp(-x * x);
                const double qq = a == 0 ? (b == 0 ? qOO : qOH) : (b == 0 ? qOH : qHH);
                const double ee = qq * (ex * erfcx(x)) * rinv;
                double df = -(ee + qq * c2a * ex) * s2;
                if (a == 0 && b == 0 && rr2 <= rv2) {
                    const double s6 = s2 * s2 * s2, A = w12 * s6 * s6, B = w6 * s6;
                    double e1 = A - B, df1 = -6.0 * s2 * (A + e1);
                    lj_switch_apply<double>(R, rr2, e1, df1);
                    e4[img ? 1 : 0] += e1;
                    e4[img ? 5 : 4] -= df1 * rr2;   // watwat_ewald_press.f:146-152
                    df += df1;
                }
                e_el += ee;
                g[3 * a] += df * dx; g[3 * a + 1] += df * dy; g[3 * a + 2] += df * dz;
                H[0] -= df * dx; H[1] -= df * dy; H[2] -= df * dz;
            }
            e4[img ? 3 : 2] += e_el;
            const size_t gj = 9 * (size_t)j + 3 * b;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (nb_below(H[d], 8)) atomicAdd(fine + gj + d, nb_fine(H[d]));
                else atomicAdd(grad + gj + d, (unsigned long long)nb_fix(H[d]));
            }
        }
        __syncwarp();
    };
    const int il = i - R.wat0;
    int cnt = 0;
    for (int k0 = 0; k0 < L1.n; k0 += 32) {
        const int k = k0 + lane;
        bool in = false, img = false;
        double dx = 0.0, dy = 0.0, dz = 0.0;
        int j = 0;
        if (k < L1.n) {
            j = L1.at(k);
            if (nb_half_owner(il, j - R.wat0) == il) {
                const double4 oj = pos[3 * (size_t)j];
                dx = oi0.x - oj.x; dy = oi0.y - oj.y; dz = oi0.z - oj.z;
                min_image(R, dx, dy, dz, img);
                in = dx * dx + dy * dy + dz * dz <= rmax2;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (cnt + __popc(m) > WBUF64) { work_off(cnt); cnt = 0; }
        if (in) {
            const int p = cnt + __popc(m & ((1u << lane) - 1u));
            D[0][p] = dx; D[1][p] = dy; D[2][p] = dz;
            J[p] = img ? ~j : j;
        }
        cnt += __popc(m);
        npair += in ? 18 : 0;
    }
    work_off(cnt);
#pragma unroll
    for (int k = 0; k < 6; ++k) e4[k] *= 2.0;   // each pair once; the energy reduction halves
    // water sites against non-water atoms (W2, full list): a lane's share of the entries
    auto none = []() {};
    water_vs_atoms(R, i, pos, lj_v, sflags, wl2_off, wl2, cap2, lane, 32, 0, g, e4, npair, none);
    bool small = true;
#pragma unroll
    for (int k = 0; k < 9; ++k) small &= nb_below(g[k], 14);
    small = __all_sync(0xffffffffu, small);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const long long v = small ? sub_sum<32>((long long)nb_fine(g[k])) : nb_fix(sub_sum<32>(g[k]));
        if (lane == k) atomicAdd((small ? fine : grad) + 9 * (size_t)i + k, (unsigned long long)v);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) e4[k] = sub_sum<32>(e4[k]);
    npair = sub_sum<32>(npair);
    if (lane == 0) {
        double *eu = e_unit + NB_EU * (size_t)i;
        eu[0] = e4[0]; eu[1] = e4[1]; eu[2] = e4[2]; eu[3] = e4[3]; eu[4] = (double)npair;
        eu[5] = 0.0; eu[6] = e4[4]; eu[7] = e4[5];
    }
}

// FP32 water exclusion corrections (cdie_ewald.f:117-199 for the pairs O-H1, O-H2, H1-H2 of
// one rigid water): the three intramolecular displacements come from the FP64-formed H
// offsets h1, h2, so no absolute FP32 coordinate enters; erf(x)/x from its Taylor series in
// u = x^2 (9 terms, truncation below 6e-9 for u <= 0.5), erff beyond.  Adds the gradient of
// the three sites to g[3 * site + axis] and returns the energy.  With R.wref the returned
// energy is the difference from the replica's reference water (wcorr0, added in FP64 by the
// energy reduction): coef * (r^2 - t0) * Q(r^2) per pair, Q the quotient of the series by
// (r^2 - t0), which keeps the FP32 error a fraction of a small difference.
__device__ __forceinline__ float water_intra_f(const RepDev &R, float4 h1, float4 h2, const float q[3], float g[9])
{
    // displacement x_a - x_b for the pairs (O,H1), (O,H2), (H1,H2)
    const float d[3][3] = {{-h1.x, -h1.y, -h1.z}, {-h2.x, -h2.y, -h2.z}, {h1.x - h2.x, h1.y - h2.y, h1.z - h2.z}};
    const int pa[3] = {0, 0, 1}, pb[3] = {1, 2, 2};
    const float al = R.alpha, ke = (float)R.epstmp, c2 = (float)NB_TWO_OVER_SQRTPI;
    float ecorr = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float rx = d[k][0], ry = d[k][1], rz = d[k][2];
        const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz)), u = al * al * r2;
        const float qq = q[pa[k]] * q[pb[k]] * ke;
        float e = 0.f, df;
        if (u <= 0.5f) {
            float ds = 8.f / 685440.f;
            ds = fmaf(ds, u, -7.f / 75600.f); ds = fmaf(ds, u, 6.f / 9360.f); ds = fmaf(ds, u, -5.f / 1320.f);
            ds = fmaf(ds, u, 4.f / 216.f); ds = fmaf(ds, u, -3.f / 42.f); ds = fmaf(ds, u, 0.2f);
            ds = fmaf(ds, u, -1.f / 3.f);
            if (!R.wref) {
                float s = 1.f / 685440.f;
                s = fmaf(s, u, -1.f / 75600.f); s = fmaf(s, u, 1.f / 9360.f); s = fmaf(s, u, -1.f / 1320.f);
                s = fmaf(s, u, 1.f / 216.f); s = fmaf(s, u, -1.f / 42.f); s = fmaf(s, u, 0.1f);
                s = fmaf(s, u, -1.f / 3.f); s = fmaf(s, u, 1.f);
                e = -qq * al * c2 * s;
            }
            df = -qq * 2.f * al * al * al * c2 * ds;
        } else {
            const float rij = sqrtf(r2), sinv = 1.f / rij, x = al * rij;
            const float erfv = erff(x), derfc = c2 * expf(-x * x);
            if (!R.wref) e = -qq * sinv * erfv;
            df = qq * sinv * (sinv * sinv * erfv - sinv * al * derfc);
        }
        if (R.wref) {
            const int ty = k == 2 ? 1 : 0;    // O-H, O-H, H-H
            float qv = R.wq[ty][7];
#pragma unroll
            for (int m = 6; m >= 0; --m) qv = fmaf(qv, r2, R.wq[ty][m]);
            e = R.wcoef[ty] * ((r2 - R.wt0[ty]) * qv);
        }
        ecorr += e;
        const int a = pa[k], b = pb[k];
        g[3 * a] += df * rx; g[3 * a + 1] += df * ry; g[3 * a + 2] += df * rz;
        g[3 * b] -= df * rx; g[3 * b + 1] -= df * ry; g[3 * b + 2] -= df * rz;
    }
    return ecorr;
}

// ---------------------------------------------------------------------------------
// FP32 water kernels on the packed two-lane FP32 pipe.
// FP32 water kernel over full rows, LPW lanes per water: the lanes take the row's entries in
// turn (consecutive lanes read consecutive entries) and each owns a partial gradient of its
// water, summed over the lanes at the end (FP32 butterfly, then fixed point).  Of an entry's nine
// site pairs eight run packed two by two on the FP32x2 pipe -- (O; H, H) and (H, H; each
// partner site) -- and the O-O pair with its LJ part runs scalar, so one partner record is
// live at a time.  Bound: for small handles the latency of a row's rounds, beyond the L1 wavefronts of
// the record gathers.  Water stage against one water per thread: 216 waters 62 -> 13 us, 7,000 79 -> 21
// (the lane counts at water_lanes).  VIR: also the water-water LJ virial terms.  ATOMS: the handle has atoms
// outside waters, whose lists (W2) come first, so that one barrier stands between the last flush of either
// list and the sums; with W2 after the rows and a barrier behind it the water stage of 28,900 waters without
// an atom took 62 us, 55 without that part, and that of 5 solute systems 129, 122 in this order.
template <int LPW, bool VIR, bool ATOMS, typename E>
__global__ void __launch_bounds__(WBLOCK, 4) k_water_s(int nW, const RepDev *__restrict__ reps,
                                                       const int *__restrict__ site_rep, const float4 *__restrict__ pos,
                                                       const float4 *__restrict__ woff, const void *lj_v,
                                                       const unsigned *__restrict__ sflags,
                                                       const int2 *__restrict__ wl1_cnt, const void *__restrict__ wl1,
                                                       int cap_row, const int *__restrict__ wl2_off,
                                                       const int *__restrict__ wl2, int cap2, long long *__restrict__ grad,
                                                       double *__restrict__ e_unit, int intra)
{
    constexpr int NE = VIR ? 6 : 4;
    __shared__ unsigned long long sG[WBLOCK / LPW][9];   // rows longer than CHUNK entries per lane
    __shared__ float2 sE[NE][WBLOCK];
    const int t = threadIdx.x, sub = t & (LPW - 1), w = t / LPW;
    const int iw = blockIdx.x * (WBLOCK / LPW) + w;
    const bool act = iw < nW;
    const int i = act ? iw : nW - 1;         // idle lanes of the last block: an empty row, no output
    const RepDev &R = reps[site_rep[3 * i]];
    for (int k = sub; k < 9; k += LPW) sG[w][k] = 0ull;
#pragma unroll
    for (int k = 0; k < NE; ++k) sE[k][t] = make_float2(0.f, 0.f);
    __syncwarp();
    const float4 oi0 = woff[3 * i], oi1 = woff[3 * i + 1], oi2 = woff[3 * i + 2];
    const float2 hx = f2(oi1.x, oi2.x), hy = f2(oi1.y, oi2.y), hz = f2(oi1.z, oi2.z);   // (H1, H2) offsets
    // minus the gradient: of O as two partials, of (H1, H2)
    float2 GO[3] = {f2(0.f), f2(0.f), f2(0.f)}, GH[3] = {f2(0.f), f2(0.f), f2(0.f)};
    float g[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) g[k] = 0.f;
    float e4[NE];    // LJ prim, LJ img, Coulomb prim, Coulomb img (, LJ virial prim, LJ virial img)
#pragma unroll
    for (int k = 0; k < NE; ++k) e4[k] = 0.f;
    auto fold = [&]() {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            g[d] -= GO[d].x + GO[d].y; g[3 + d] -= GH[d].x; g[6 + d] -= GH[d].y;
            GO[d] = f2(0.f); GH[d] = f2(0.f);
        }
    };
    auto flush_e = [&]() {
#pragma unroll
        for (int k = 0; k < NE; ++k) { two_add(sE[k][t], e4[k]); e4[k] = 0.f; }
    };
    auto flush_all = [&]() {
        fold();
#pragma unroll
        for (int k = 0; k < 9; ++k) { atomicAdd(&sG[w][k], (unsigned long long)nb_fix(g[k])); g[k] = 0.f; }
        flush_e();
    };
    int npair = 0;
    const float iL0 = held(R.invL[0]), iL1 = held(R.invL[1]), iL2 = held(R.invL[2]);
    const float L0 = held(R.L[0]), L1 = held(R.L[1]), L2 = held(R.L[2]);
    const float m0 = held(R.Llo[0]), m1 = held(R.Llo[1]), m2 = held(R.Llo[2]);
    const float rmax2 = held(R.rmax2), rv2 = held(R.rv2);
    const WaterK K = {held(ERFCX_P * R.alpha), held(R.ex2c), held(R.c2a)};
    const float qOO = held(R.qq[0]), qOH = held(R.qq[1]), qHH = held(R.qq[2]), w12 = held(R.w12), w6 = held(R.w6);
    const float w12c = held(R.w12c), w6c = held(R.w6c);
    const bool sw = R.lj_switch != 0;
    const W1Row<E> row(wl1_cnt, wl1, cap_row, i, R.wat0);
    const int n = act ? row.n : 0;
    // one molecule pair: the partner's record (O, then the H offsets)
    auto pair = [&](float4 oj, float4 a, float4 b) {
        float dx = oi0.x - oj.x, dy = oi0.y - oj.y, dz = oi0.z - oj.z;
        // (x + 1.5*2^23) - 1.5*2^23 rounds x to nearest (|x| < 2^22)
        const float nx = fmaf(dx, iL0, 12582912.f) - 12582912.f, ny = fmaf(dy, iL1, 12582912.f) - 12582912.f,
                    nz = fmaf(dz, iL2, 12582912.f) - 12582912.f;
        dx = fmaf(-nx, m0, fmaf(-nx, L0, dx)); dy = fmaf(-ny, m1, fmaf(-ny, L1, dy)); dz = fmaf(-nz, m2, fmaf(-nz, L2, dz));
        const float r2 = dx * dx + dy * dy + dz * dz;
        if (r2 <= rmax2) {
            float2 eel, e;
            float eoo, elj = 0.f, vlj = 0.f;
            {
                // O-O: Coulomb and LJ (powers from a Newton-refined 1/r: r^-12 amplifies the
                // approximate rsqrt's error 12 times; the correction is formed as a small number)
                const float rr2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                const float rinv = nb_rsqrt_approx(rr2), s2 = rinv * rinv;
                float mdf = ewald1(K, rr2, rinv, qOO, eoo);
                if (rr2 <= rv2) {
                    const float ri = fmaf(-0.5f * rinv, fmaf(rr2, s2, -1.f), rinv), sl = ri * ri;
                    const float s6 = sl * sl * sl, A = w12 * s6 * s6;
                    // c12, c6 restore the FP32 rounding of the coefficients in the energy (the force
                    // keeps A and B)
                    float e1 = fmaf(-w6, fmaf(s6, w6c, s6), fmaf(A, w12c, A));
                    float m1 = 6.f * sl * fmaf(-w6, s6, A + A);
                    if (sw) {
                        float d1 = -m1;
                        lj_switch_apply<float>(R, rr2, e1, d1);
                        m1 = -d1;
                    }
                    elj = e1;
                    if (VIR) vlj = m1 * rr2;   // -df1 r^2 (watwat_ewald_press.f:146-152)
                    mdf += m1;
                }
                GO[0].x = fmaf(mdf, dx, GO[0].x); GO[1].x = fmaf(mdf, dy, GO[1].x); GO[2].x = fmaf(mdf, dz, GO[2].x);
            }
            {
                // O of i with (H1, H2) of j
                const float2 x = f2(dx - a.x, dx - b.x), y = f2(dy - a.y, dy - b.y), z = f2(dz - a.z, dz - b.z);
                const float2 m = ewald2(K, __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z))), f2(qOH), eel);
                GO[0] = __ffma2_rn(m, x, GO[0]); GO[1] = __ffma2_rn(m, y, GO[1]); GO[2] = __ffma2_rn(m, z, GO[2]);
            }
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                // (H1, H2) of i with site s of j
                const float qx = s == 0 ? dx : (s == 1 ? dx - a.x : dx - b.x);
                const float qy = s == 0 ? dy : (s == 1 ? dy - a.y : dy - b.y);
                const float qz = s == 0 ? dz : (s == 1 ? dz - a.z : dz - b.z);
                const float2 x = __fadd2_rn(hx, f2(qx)), y = __fadd2_rn(hy, f2(qy)), z = __fadd2_rn(hz, f2(qz));
                const float2 m = ewald2(K, __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z))),
                                        f2(s == 0 ? qOH : qHH), e);
                eel = __fadd2_rn(eel, e);
                GH[0] = __ffma2_rn(m, x, GH[0]); GH[1] = __ffma2_rn(m, y, GH[1]); GH[2] = __ffma2_rn(m, z, GH[2]);
            }
            const bool img = (nx != 0.f) | (ny != 0.f) | (nz != 0.f);
            const float ec = eoo + (eel.x + eel.y);
            e4[0] += img ? 0.f : elj; e4[1] += img ? elj : 0.f;
            e4[2] += img ? 0.f : ec; e4[3] += img ? ec : 0.f;
            if (VIR) { e4[NE - 2] += img ? 0.f : vlj; e4[NE - 1] += img ? vlj : 0.f; }
            npair += 9;
        }
    };
    int cnt = 0;
    if constexpr (ATOMS) {
        if (act) {
            const AtomK A(R, iL0, iL1, iL2, L0, L1, L2, m0, m1, m2, rmax2, rv2, K);
            water_vs_atoms(R, A, i, pos, lj_v, sflags, wl2_off, wl2, cap2, sub, LPW, cnt, g, e4, npair, flush_all);
        }
        __syncwarp();
    }
    // two record buffers in turn, as in k_water_h: the next entry's record is on its way while one is
    // worked on, row entries two ahead of their records
    if (sub < n) {
        auto entry = [&](int k) { return row.at(min(k, n - 1)); };
        int ja = entry(sub), jb = entry(sub + LPW);
        const float4 *r = woff + 3 * (size_t)ja;
        float4 oa = r[0], ha = r[1], ia = r[2];
        for (int k = sub; k < n; k += 2 * LPW) {
            const int jc = entry(k + 2 * LPW), jd = entry(k + 3 * LPW);
            r = woff + 3 * (size_t)jb;
            const float4 ob = r[0], hb = r[1], ib = r[2];
            pair(oa, ha, ia);
            r = woff + 3 * (size_t)jc;
            oa = r[0]; ha = r[1]; ia = r[2];
            if (k + LPW < n) pair(ob, hb, ib);
            jb = jd;
            cnt += 2;
            if (cnt >= CHUNK - 1) { flush_all(); cnt = 0; }     // (64 entries; 63 or 64 behind a list of atoms)
        }
    }
    // rows differ in length: the lanes that end early wait here, and the last flushes into sG come before
    // its reads (the shuffles below order no memory)
    __syncwarp();
    fold();
    // the molecule's own exclusion corrections (every water excludes exactly its three pairs), in every lane; as
    // large as all its other forces together, they join them after the sum over the lanes (a fixed-point
    // number of their own cost 5 us of 28,900 waters' evaluation: conversions to 64 bits take the FP64 pipe)
    float ecorr = 0.f, gi[9] = {};
    if (intra) {
        const float qs[3] = {oi0.w, oi1.w, oi2.w};
        ecorr = water_intra_f(R, oi1, oi2, qs, gi);
    }
    flush_e();
#pragma unroll
    for (int k = 0; k < 9; ++k)
#pragma unroll
        for (int o = LPW / 2; o > 0; o >>= 1) g[k] += __shfl_xor_sync(0xffffffffu, g[k], o, LPW);
    npair = sub_sum<LPW>(npair);
    float2 es[NE];
#pragma unroll
    for (int k = 0; k < NE; ++k) es[k] = sub_two_sum<LPW>(sE[k][t]);
    if (!act) return;
#pragma unroll
    for (int k = 0; k < 9; ++k)
        if (sub == k % LPW) grad[(size_t)9 * i + k] = nb_fix(g[k] + gi[k]) + (long long)sG[w][k];
    if (sub == 0) {
        double *eu = e_unit + NB_EU * (size_t)i;
#pragma unroll
        for (int k = 0; k < 4; ++k) eu[k] = (double)es[k].x + (double)es[k].y;
        eu[4] = (double)npair;
        eu[5] = (double)ecorr;
        eu[6] = VIR ? (double)es[NE - 2].x + (double)es[NE - 2].y : 0.0;
        eu[7] = VIR ? (double)es[NE - 1].x + (double)es[NE - 1].y : 0.0;
    }
}

// ---------------------------------------------------------------------------------
// FP32 water kernel over half lists (k_whalf): every water-water pair is evaluated once, by
// its owner, with the pair arithmetic of k_water_s (eight of the nine site pairs packed two by
// two).  One water per thread, whose gradient stays in registers; the partner's side of each
// pair goes to an int32 accumulator in shared memory indexed by the partner's place in the
// block's j-set, at 2^S units per kcal/mol/Å (S = 24 - log2 HB).  A share is rounded to the unit by
// adding 1.5 * 2^23 (a conversion would share the special-function pipe with rsqrt, rcp and
// ex2), so it has to stay below 2^22 units, and HB of those cannot overflow; larger shares go
// directly to the int64 gradient.  At the end the block adds its j-set sums and its own waters'
// gradients to the int64 site gradient with atomics (integer sums: the result does not depend
// on their order).  The site gradient of the waters is cleared before the launch.  Water-water
// energies and pair counts are doubled, as the energy reduction halves the full-list sums.
// Bound: instruction issue at the 16 warps that 128 registers allow, then the latency of the
// partner gathers.  Two list entries per iteration packed on the FP32x2 pipe left 4 warps in 10
// waiting for gathers (issue 35%): the hydrogens' loads depended on the O-O test, and lanes with
// short rows ran the flush apart from the others.  Water stage, 256 replicas (433,195 waters):
// 625 us; whole records one entry ahead and constants held in registers 543; the lanes together
// before the tail, one gradient flush per row, loads without a branch 513; two record buffers in
// turn 490; the rounding by addition 482.  A thread's gradient and energies are flushed every CHUNK
// entries (every 128: the evaluation of 32,000 waters 1% shorter, its gradient's error in FP32's rounding
// 0.01% larger; two accumulators per hydrogen: no smaller).  Records staged in shared memory per block (a warp per
// water, lanes over its row) took 50% more instructions and 750 us.
template <int HB> struct HalfScale;
template <> struct HalfScale<128> { static constexpr int S = 17; };
template <> struct HalfScale<256> { static constexpr int S = 16; };
template <> struct HalfScale<512> { static constexpr int S = 15; };

// VIR: also the water-water LJ virial terms (as k_water_s<.., true, ..>)
template <int HB, bool VIR>
__global__ void __launch_bounds__(HB, 512 / HB) k_water_h(const int2 *__restrict__ blocks, const RepDev *__restrict__ reps,
                                                          const float4 *__restrict__ pos, const float4 *__restrict__ woff,
                                                          const void *lj_v, const unsigned *__restrict__ sflags,
                                                          const unsigned *__restrict__ hrow, int caph,
                                                          const int2 *__restrict__ hcnt, const int *__restrict__ jset,
                                                          const int *__restrict__ jn, int jcap, int jsh,
                                                          const int *__restrict__ wl2_off, const int *__restrict__ wl2,
                                                          int cap2, long long *__restrict__ grad,
                                                          double *__restrict__ e_unit, int intra)
{
    constexpr int S = HalfScale<HB>::S;
    constexpr float SC = (float)(1 << S), CAP = 4.19e6f / SC;   // (2^22 = 4,194,304)
    constexpr int NE = VIR ? 6 : 4;
    __shared__ float2 sE[NE][HB];
    extern __shared__ int sJ[];      // [9][jsh]: partner-site gradients, 2^S units
    const int t = threadIdx.x, b = blockIdx.x;
    const int2 w = blocks[b];
    const RepDev &R = reps[w.x];
    const int nJ = min(jn[b], jsh);
    for (int k = t; k < nJ; k += HB)
#pragma unroll
        for (int c = 0; c < 9; ++c) sJ[c * jsh + k] = 0;
#pragma unroll
    for (int k = 0; k < NE; ++k) sE[k][t] = make_float2(0.f, 0.f);
    __syncthreads();
    const int i = w.y + t;
    const unsigned present = __ballot_sync(0xffffffffu, i - R.wat0 < R.nwat);
    if (i - R.wat0 < R.nwat) {
        const float4 oi0 = woff[3 * i];
        const float4 oi1 = woff[3 * i + 1], oi2 = woff[3 * i + 2];
        const float2 hx = f2(oi1.x, oi2.x), hy = f2(oi1.y, oi2.y), hz = f2(oi1.z, oi2.z);   // (H1, H2) offsets
        // minus the gradient: of O as two partials, of (H1, H2)
        float2 GO[3] = {f2(0.f), f2(0.f), f2(0.f)}, GH[3] = {f2(0.f), f2(0.f), f2(0.f)};
        // the owner's gradient goes to the int64 site gradient with one atomic per component
        // and flush (no shared-memory slots: they would take the L1 that the gathers use)
        unsigned long long *gi = (unsigned long long *)(grad + 9 * (size_t)i);
        float g[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) g[k] = 0.f;
        // LJ prim, LJ img, Coulomb prim, Coulomb img (, LJ virial prim, LJ virial img)
        float e4[NE];
#pragma unroll
        for (int k = 0; k < NE; ++k) e4[k] = 0.f;
        double *eu = e_unit + NB_EU * (size_t)i;
        // ef: 2 for the water-water energies (each pair once), 1 for the W2 part (full list); gi9: a gradient
        // rounded to fixed point by itself
        auto flush = [&](float ef, const float *gi9) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                g[d] -= GO[d].x + GO[d].y; g[3 + d] -= GH[d].x; g[6 + d] -= GH[d].y;
                GO[d] = f2(0.f); GH[d] = f2(0.f);
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const long long v = nb_fix(g[k]) + (gi9 ? nb_fix(gi9[k]) : 0LL);
                if (v != 0) atomicAdd(gi + k, (unsigned long long)v);
                g[k] = 0.f;
            }
#pragma unroll
            for (int k = 0; k < NE; ++k) { two_add(sE[k][t], ef * e4[k]); e4[k] = 0.f; }
        };
        auto flush1 = [&]() { flush(1.f, nullptr); };
        int npair = 0;
        const float iL0 = held(R.invL[0]), iL1 = held(R.invL[1]), iL2 = held(R.invL[2]);
        const float rmax2 = held(R.rmax2), rv2 = held(R.rv2);
        const WaterK K = {held(ERFCX_P * R.alpha), held(R.ex2c), held(R.c2a)};
        const float qOO = held(R.qq[0]), qOH = held(R.qq[1]), qHH = held(R.qq[2]), w12 = held(R.w12), w6 = held(R.w6);
        const float w12c = held(R.w12c), w6c = held(R.w6c);
        const float L0 = held(R.L[0]), L1 = held(R.L[1]), L2 = held(R.L[2]);
        const float m0 = held(R.Llo[0]), m1 = held(R.Llo[1]), m2 = held(R.Llo[2]);
        const bool sw = held(__int_as_float(R.lj_switch)) != 0.f;
        const unsigned *hr = hrow + (size_t)b * caph * HB + t;
        const int k1 = hcnt[i].y, wat0 = R.wat0;
        int cnt = 0;
        // one molecule pair: entry en, the partner's record
        auto pair = [&](unsigned en, float4 oj, float4 A, float4 B) {
            float dx = oi0.x - oj.x, dy = oi0.y - oj.y, dz = oi0.z - oj.z;
            const float nx = fmaf(dx, iL0, 12582912.f) - 12582912.f, ny = fmaf(dy, iL1, 12582912.f) - 12582912.f,
                        nz = fmaf(dz, iL2, 12582912.f) - 12582912.f;
            dx = fmaf(-nx, m0, fmaf(-nx, L0, dx)); dy = fmaf(-ny, m1, fmaf(-ny, L1, dy)); dz = fmaf(-nz, m2, fmaf(-nz, L2, dz));
            if (dx * dx + dy * dy + dz * dz <= rmax2) {
                float H[9];      // the partner's gradient
                float2 eel, e;
                float eoo, elj = 0.f, vlj = 0.f;
                {
                    // O-O: Coulomb and LJ, as k_water_s
                    const float rr2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                    const float rinv = nb_rsqrt_approx(rr2), s2 = rinv * rinv;
                    float mdf = ewald1(K, rr2, rinv, qOO, eoo);
                    if (rr2 <= rv2) {
                        const float ri = fmaf(-0.5f * rinv, fmaf(rr2, s2, -1.f), rinv), sl = ri * ri;
                        const float s6 = sl * sl * sl, LA = w12 * s6 * s6;
                        float e1 = fmaf(-w6, fmaf(s6, w6c, s6), fmaf(LA, w12c, LA));
                        float m1 = 6.f * sl * fmaf(-w6, s6, LA + LA);
                        if (sw) {
                            float d1 = -m1;
                            lj_switch_apply<float>(R, rr2, e1, d1);
                            m1 = -d1;
                        }
                        elj = e1;
                        if (VIR) vlj = m1 * rr2;   // -df1 r^2 (watwat_ewald_press.f:146-152)
                        mdf += m1;
                    }
                    H[0] = mdf * dx; H[1] = mdf * dy; H[2] = mdf * dz;
                    GO[0].x += H[0]; GO[1].x += H[1]; GO[2].x += H[2];
                }
                const float ax = dx - A.x, ay = dy - A.y, az = dz - A.z, bx = dx - B.x, by = dy - B.y, bz = dz - B.z;
                {
                    // O of i with (H1, H2) of j
                    const float2 x = f2(ax, bx), y = f2(ay, by), z = f2(az, bz);
                    const float2 m = ewald2(K, __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z))), f2(qOH), eel);
                    const float2 fx = __fmul2_rn(m, x), fy = __fmul2_rn(m, y), fz = __fmul2_rn(m, z);
                    GO[0] = __fadd2_rn(GO[0], fx); GO[1] = __fadd2_rn(GO[1], fy); GO[2] = __fadd2_rn(GO[2], fz);
                    H[3] = fx.x; H[4] = fy.x; H[5] = fz.x;
                    H[6] = fx.y; H[7] = fy.y; H[8] = fz.y;
                }
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    // (H1, H2) of i with site s of j
                    const float2 x = __fadd2_rn(hx, f2(s == 0 ? dx : (s == 1 ? ax : bx)));
                    const float2 y = __fadd2_rn(hy, f2(s == 0 ? dy : (s == 1 ? ay : by)));
                    const float2 z = __fadd2_rn(hz, f2(s == 0 ? dz : (s == 1 ? az : bz)));
                    const float2 m = ewald2(K, __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z))),
                                            f2(s == 0 ? qOH : qHH), e);
                    eel = __fadd2_rn(eel, e);
                    const float2 fx = __fmul2_rn(m, x), fy = __fmul2_rn(m, y), fz = __fmul2_rn(m, z);
                    GH[0] = __fadd2_rn(GH[0], fx); GH[1] = __fadd2_rn(GH[1], fy); GH[2] = __fadd2_rn(GH[2], fz);
                    H[3 * s] += fx.x + fx.y; H[3 * s + 1] += fy.x + fy.y; H[3 * s + 2] += fz.x + fz.y;
                }
                const int l = (int)(en >> 16);
                float hm = 0.f;
#pragma unroll
                for (int c = 0; c < 9; ++c) hm = fmaxf(hm, fabsf(H[c]));
                if (hm < CAP && l < jsh) {
#pragma unroll
                    for (int c = 0; c < 9; ++c)
                        atomicAdd(&sJ[c * jsh + l], __float_as_int(fmaf(H[c], SC, 12582912.f)) - 0x4b400000);
                } else {
                    // a large share (rare), or a partner past the shared memory: to the int64 gradient
                    unsigned long long *gj = (unsigned long long *)(grad + 9 * (size_t)(wat0 + (int)(en & 0xffffu)));
#pragma unroll
                    for (int c = 0; c < 9; ++c) atomicAdd(gj + c, (unsigned long long)nb_fix(H[c]));
                }
                const bool img = (nx != 0.f) | (ny != 0.f) | (nz != 0.f);
                const float ec = eoo + (eel.x + eel.y);
                e4[0] += img ? 0.f : elj; e4[1] += img ? elj : 0.f;
                e4[2] += img ? 0.f : ec; e4[3] += img ? ec : 0.f;
                if (VIR) { e4[NE - 2] += img ? 0.f : vlj; e4[NE - 1] += img ? vlj : 0.f; }
                npair += 18;
            }
        };
        // The next entry's record is on its way while one is worked on: two record buffers in turn
        // (a copy between them would tie a load to the end of the previous use of its registers),
        // row entries two ahead of their records, the warp's row lines (one 128-byte line per
        // entry) in L1 eight ahead.
        auto rec = [&](unsigned en) { return woff + 3 * (wat0 + (int)(en & 0xffffu)); };
        auto entry = [&](int k) { return hr[(size_t)min(k, k1 - 1) * HB]; };
        if (k1 > 0) {
            unsigned ea = entry(0), eb = entry(1);
            const float4 *r = rec(ea);
            float4 oa = r[0], ha = r[1], ia = r[2];
            for (int k = 0; k < k1; k += 2) {
                const unsigned ec = entry(k + 2), ed = entry(k + 3);
                r = rec(eb);
                const float4 ob = r[0], hb = r[1], ib = r[2];
                nb_prefetch_l1(hr + (size_t)min(k + 8, k1 - 1) * HB);
                nb_prefetch_l1(hr + (size_t)min(k + 9, k1 - 1) * HB);
                pair(ea, oa, ha, ia);
                r = rec(ec);
                oa = r[0]; ha = r[1]; ia = r[2];
                if (k + 1 < k1) pair(eb, ob, hb, ib);
                ea = ec; eb = ed;
                cnt += 2;
                if (cnt >= CHUNK) { flush(2.f, nullptr); cnt = 0; }
            }
        }
        __syncwarp(present);     // rows differ in length: without this, lanes that end early run the tail apart
        // the molecule's own exclusion corrections join the last flush, as numbers of their own (k_water_s)
        float ecorr = 0.f, gx[9] = {};
        if (intra) {
            const float4 w1 = woff[3 * i + 1], w2 = woff[3 * i + 2];
            const float qs[3] = {oi0.w, w1.w, w2.w};
            ecorr = water_intra_f(R, w1, w2, qs, gx);
        }
        eu[5] = (double)ecorr;
        flush(2.f, gx);
        if (wl2_off[i] < wl2_off[i + 1]) {
            const AtomK A(R, iL0, iL1, iL2, L0, L1, L2, m0, m1, m2, rmax2, rv2, K);
            cnt = 0;
            water_vs_atoms(R, A, i, pos, lj_v, sflags, wl2_off, wl2, cap2, 0, 1, cnt, g, e4, npair, flush1);
            flush1();
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) eu[k] = (double)sE[k][t].x + (double)sE[k][t].y;
        eu[4] = (double)npair;
        eu[6] = VIR ? (double)sE[NE - 2][t].x + (double)sE[NE - 2][t].y : 0.0;
        eu[7] = VIR ? (double)sE[NE - 1][t].x + (double)sE[NE - 1][t].y : 0.0;
    }
    __syncthreads();
    // the block's partner shares of its j-set: a warp takes 32 partners, and its lanes the 288
    // words of their gradients in order (nine consecutive words per partner, so a request
    // touches 9 sectors instead of 32)
    const int *js = jset + (size_t)b * jcap;
    const int lane = t & 31;
    for (int l0 = t - lane; l0 < nJ; l0 += HB) {
        const int jl = l0 + lane < nJ ? js[l0 + lane] : -1;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int f = 32 * q + lane, l = f / 9, c = f - 9 * l;
            const int j = __shfl_sync(0xffffffffu, jl, l);
            const int v = j >= 0 ? sJ[c * jsh + l0 + l] : 0;
            if (v != 0) atomicAdd((unsigned long long *)&grad[9 * (size_t)j + c], (unsigned long long)((long long)v * (1LL << (32 - S))));
        }
    }
}

// One warp per non-water atom over its full site list: the lanes take the list's entries in turn
// (consecutive entries are mostly the sites of one water, so the position loads coalesce) and
// their partial gradients and energies are summed over the warp at the end; every pair's energies and LJ
// virial go into hi + lo pairs (two_add2).  One atom per thread ran its ~600 entries in series: 486 us for 2,496 atoms, 363 us for
// 203.  Bound: instruction issue; with the constants loaded again for every pair and six hi + lo
// sums per pair 19,968 atoms took 90 us, with held constants, records one entry ahead, six blocks per
// multiprocessor and the sums two at once 71 (68 with FP32 sums of 16 pairs between).
#define CHUNK_ATOM 16
__global__ void __launch_bounds__(128, 6) k_atom_f(int nA, int nW, const RepDev *__restrict__ reps,
                                                const int *__restrict__ site_rep, const float4 *__restrict__ pos,
                                                const float2 *__restrict__ lj, const unsigned *__restrict__ sflags,
                                                const int *__restrict__ xl_off, const int *__restrict__ xl, int capx,
                                                long long *__restrict__ grad, double *__restrict__ e_unit)
{
    const int lane = threadIdx.x & 31, k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= nA) return;
    const int si = 3 * nW + k;
    const RepDev &R = reps[site_rep[si]];
    const AtomK A(R);
    const float4 xi = pos[si];
    const float2 lji = lj[si];
    const float qi = xi.w * A.ke;
    const unsigned fi = A.tiny ? sflags[si] & SF_HTINY : 0;
    float g[3] = {0.f, 0.f, 0.f};
    long long G[3] = {0, 0, 0};
    float2 eh[3], el[3];     // LJ, Coulomb and LJ virial, (primary box, images): hi and lo
#pragma unroll
    for (int m = 0; m < 3; ++m) { eh[m] = f2(0.f); el[m] = f2(0.f); }
    int cnt = 0, npair = 0;
    // an overflowed list is read within the buffer (the evaluation is redone)
    const int q0 = min(xl_off[k], capx), q1 = min(xl_off[k + 1], capx);
    if (q0 + lane < q1) {
        // the next entry's record is on its way while one is worked on, its index one further ahead
        auto entry = [&](int q) { return xl[min(q, q1 - 1)]; };
        int s = entry(q0 + lane), sn = entry(q0 + lane + 32);
        float4 xj = pos[s];
        float2 ljj = lj[s];
        for (int q = q0 + lane; q < q1; q += 32) {
            const int sc = s;
            const float4 xc = xj;
            const float2 lc = ljj;
            s = sn;
            xj = pos[s]; ljj = lj[s];
            sn = entry(q + 64);
            float dx = xi.x - xc.x, dy = xi.y - xc.y, dz = xi.z - xc.z;
            bool img;
            A.image(dx, dy, dz, img);
            const bool t = A.tiny && ((fi | (sflags[sc] & SF_HTINY)) != 0);
            float eel, elj, vir;
            const float m = A.pair(R, dx * dx + dy * dy + dz * dz, qi * xc.w, lji, lc, t, eel, elj, vir, npair);
            g[0] = fmaf(-m, dx, g[0]); g[1] = fmaf(-m, dy, g[1]); g[2] = fmaf(-m, dz, g[2]);
            // LJ virial: a water partner's side of the pair (its W2 list) adds none, so it counts
            // twice here; pairs of two non-water atoms are seen from both sides
            if (sc < 3 * nW) vir += vir;
            two_add2(eh[0], el[0], f2(img ? 0.f : elj, img ? elj : 0.f));
            two_add2(eh[1], el[1], f2(img ? 0.f : eel, img ? eel : 0.f));
            two_add2(eh[2], el[2], f2(img ? 0.f : vir, img ? vir : 0.f));
            if (++cnt == CHUNK_ATOM) { flush(g, G, 3); cnt = 0; }
        }
    }
    __syncwarp();
    flush(g, G, 3);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const long long v = sub_sum<32>(G[d]);
        if (lane == d) grad[(size_t)3 * si + d] = v;
    }
    double e[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const float2 v = sub_two_sum<32>(m & 1 ? f2(eh[m / 2].y, el[m / 2].y) : f2(eh[m / 2].x, el[m / 2].x));
        e[m] = (double)v.x + (double)v.y;
    }
    npair = sub_sum<32>(npair);
    if (lane == 0) {
        double *eu = e_unit + NB_EU * (size_t)(nW + k);
        eu[0] = e[0]; eu[1] = e[1]; eu[2] = e[2]; eu[3] = e[3]; eu[4] = (double)npair; eu[5] = 0.0;
        eu[6] = e[4]; eu[7] = e[5];
    }
}

// The same on the plain FP64 path
__global__ void __launch_bounds__(128) k_atom_d(int nA, int nW, const RepDev *__restrict__ reps, const int *__restrict__ site_rep,
                                              const void *pos_v, const void *lj_v, const unsigned *__restrict__ sflags,
                                              const int *__restrict__ xl_off, const int *__restrict__ xl, int capx,
                                              long long *__restrict__ grad, double *__restrict__ e_unit)
{
    const int lane = threadIdx.x & 31, k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= nA) return;
    typedef double T;
    typedef double4 T4;
    typedef double2 T2;
    const T4 *pos = (const T4 *)pos_v;
    const T2 *lj = (const T2 *)lj_v;
    int si = 3 * nW + k;
    const RepDev &R = reps[site_rep[si]];
    T4 xi = pos[si];
    T2 lji = lj[si];
    unsigned fi = sflags[si];
    T g[3] = {0, 0, 0};
    T es[6] = {0, 0, 0, 0, 0, 0};    // LJ prim, LJ img, Coulomb prim, Coulomb img, LJ virial prim, img
    int npair = 0;
    // an overflowed list is read within the buffer (the evaluation is redone)
    const int q1 = min(xl_off[k + 1], capx);
    for (int q = min(xl_off[k], capx) + lane; q < q1; q += 32) {
        int s = xl[q];
        T4 xj = pos[s];
        T2 ljj = lj[s];
        T dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        bool img;
        min_image(R, dx, dy, dz, img);
        T r2 = dx * dx + dy * dy + dz * dz;
        T eel = 0, elj = 0, vir = 0;
        T df = atom_pair(R, r2, xi.w, xj.w, lji.x, lji.y, ljj.x, ljj.y, fi, sflags[s], eel, elj, vir, npair);
        g[0] += df * dx; g[1] += df * dy; g[2] += df * dz;
        // LJ virial: a water partner's side of the pair (its W2 list) adds none, so it counts
        // twice here; pairs of two non-water atoms are seen from both sides
        if (s < 3 * nW) vir += vir;
        es[0] += img ? (T)0 : elj; es[1] += img ? elj : (T)0;
        es[2] += img ? (T)0 : eel; es[3] += img ? eel : (T)0;
        es[4] += img ? (T)0 : vir; es[5] += img ? vir : (T)0;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double v = sub_sum<32>(g[d]);
        if (lane == d) grad[(size_t)3 * si + d] = nb_fix(v);
    }
    double e[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) e[m] = sub_sum<32>(es[m]);
    npair = sub_sum<32>(npair);
    if (lane == 0) {
        double *eu = e_unit + NB_EU * (size_t)(nW + k);
        eu[0] = e[0]; eu[1] = e[1]; eu[2] = e[2]; eu[3] = e[3]; eu[4] = (double)npair; eu[5] = 0.0;
        eu[6] = e[4]; eu[7] = e[5];
    }
}

// ---------------------------------------------------------------------------------
// Water exclusion corrections (cdie_ewald.f:117-199 for the O-H1, O-H2, H1-H2 pairs of each
// water), one thread per molecule, each pair once.  With u = (alpha r)^2,
//   e  = -qq erf(alpha r)/r = -qq alpha (2/sqrt(pi)) S(u),   S(u) = sum (-1)^n u^n / (n! (2n+1))
//   df = (de/dr)/r          = -qq (4 alpha^3/sqrt(pi)) S'(u)
// (Taylor series of erf, Abramowitz & Stegun 7.1.5), evaluated in FP64 with 16 terms, which
// is exact to rounding for u <= 0.5 (r <= 2.0 Å at alpha 0.35); larger u uses erf/exp.
__constant__ double c_erf_s[16] = {
    1, -0.33333333333333331, 0.10000000000000001, -0.023809523809523808, 0.0046296296296296294,
    -0.00075757575757575758, 0.00010683760683760684, -1.3227513227513228e-05, 1.4589169000933706e-06,
    -1.4503852223150468e-07, 1.3122532963802806e-08, -1.0892221037148573e-09, 8.3507027951472397e-11,
    -5.9477940136376354e-12, 3.9554295164585257e-13, -2.4668270102644571e-14};
__constant__ double c_erf_ds[15] = {
    -0.33333333333333331, 0.20000000000000001, -0.071428571428571425, 0.018518518518518517,
    -0.003787878787878788, 0.00064102564102564103, -9.2592592592592588e-05, 1.1671335200746965e-05,
    -1.3053467000835422e-06, 1.3122532963802806e-07, -1.1981443140863431e-08, 1.0020843354176688e-09,
    -7.7321322177289257e-11, 5.537601323041936e-12, -3.7002405153966856e-13};

__device__ __forceinline__ void excl_pair(double qq, double al, double rx, double ry, double rz, double &e, double &df)
{
    double r2 = rx * rx + ry * ry + rz * rz, u = al * al * r2;
    if (u <= 0.5) {
        double s = c_erf_s[15], ds = c_erf_ds[14];
#pragma unroll
        for (int k = 14; k >= 0; --k) s = fma(s, u, c_erf_s[k]);
#pragma unroll
        for (int k = 13; k >= 0; --k) ds = fma(ds, u, c_erf_ds[k]);
        e = -qq * al * NB_TWO_OVER_SQRTPI * s;
        df = -qq * 2.0 * al * al * al * NB_TWO_OVER_SQRTPI * ds;
    } else {
        double rij = sqrt(r2), sinv = 1.0 / rij, x = al * rij;
        double erfv = erf(x), derfc = NB_TWO_OVER_SQRTPI * exp(-x * x);
        e = -qq * sinv * erfv;
        df = qq * sinv * (sinv * sinv * erfv - sinv * al * derfc);
    }
}

__global__ void k_excl_water(int nW, const int *__restrict__ unit_atom, const int *__restrict__ atom_rep,
                             const RepDev *__restrict__ reps, const double *__restrict__ coor,
                             const double *__restrict__ q, double *__restrict__ grad, double *__restrict__ e_out)
{
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nW) return;
    const int a0 = unit_atom[u];
    const RepDev &R = reps[atom_rep[a0]];
    double x[3][3], qs[3], g[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, ecorr = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        x[k][0] = coor[3 * (size_t)(a0 + k)];
        x[k][1] = coor[3 * (size_t)(a0 + k) + 1];
        x[k][2] = coor[3 * (size_t)(a0 + k) + 2];
        qs[k] = q[a0 + k];
    }
    const int pa[3] = {0, 0, 1}, pb[3] = {1, 2, 2};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const int a = pa[p], b = pb[p];
        double rx = x[a][0] - x[b][0], ry = x[a][1] - x[b][1], rz = x[a][2] - x[b][2];
        double e, df;
        excl_pair(qs[a] * qs[b] * R.epstmp, R.alphad, rx, ry, rz, e, df);
        ecorr += e;
        g[a][0] += df * rx; g[a][1] += df * ry; g[a][2] += df * rz;
        g[b][0] -= df * rx; g[b][1] -= df * ry; g[b][2] -= df * rz;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double *gp = grad + 3 * (size_t)(a0 + k), *ep = e_out + NB_EX * (size_t)(a0 + k);
        gp[0] = g[k][0]; gp[1] = g[k][1]; gp[2] = g[k][2];
        ep[0] = k == 0 ? ecorr : 0.0; ep[1] = 0.0; ep[2] = 0.0; ep[3] = 0.0;
    }
}

// exclusion erf corrections (cdie_ewald.f:117-199) and 1-4 terms (ener14.f:38-95), FP64,
// gathered per atom over both directions; raw (unimaged) displacements as MOIL uses.  Eight
// lanes per atom share its exclusions and 1-4 pairs (an erf, exp, square root and division in
// FP64 each: one atom per thread ran about eight in series, 33 us whatever the system's size), in
// blocks of one warp, which spread the FP64 work evenly over the multiprocessors (2,496 atoms: blocks
// of 128 16.5 us, 12.4).
// atoms: the n atoms to take (NULL: atom k itself); those left out belong to k_excl_water or
// the FP32 water kernels.
#define EX_LANES 8
__global__ void k_excl14(int n, const int *__restrict__ atoms, const int *__restrict__ atom_rep, const RepDev *__restrict__ reps,
                         const double *__restrict__ coor, const double *__restrict__ q, const int *__restrict__ ex_off,
                         const int *__restrict__ ex_j, const int *__restrict__ p_off, const int *__restrict__ p_j,
                         const double *__restrict__ p_par, int fixed_out, double *__restrict__ grad,
                         double *__restrict__ e_out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, sub = t & (EX_LANES - 1), u = t / EX_LANES;
    const bool act = u < n;
    const int a = act ? (atoms ? atoms[u] : u) : 0;
    const RepDev &R = reps[atom_rep[a]];
    double xa = coor[3 * (size_t)a], ya = coor[3 * (size_t)a + 1], za = coor[3 * (size_t)a + 2];
    double gx = 0, gy = 0, gz = 0, ecorr = 0, eel14 = 0, evdw14 = 0, vir14 = 0;
    double qa = q[a] * R.epstmp, al = R.alphad;
    for (int k = ex_off[a] + sub; act && k < ex_off[a + 1]; k += EX_LANES) {
        int b = ex_j[k];
        double rx = xa - coor[3 * (size_t)b], ry = ya - coor[3 * (size_t)b + 1], rz = za - coor[3 * (size_t)b + 2];
        double r2 = rx * rx + ry * ry + rz * rz, s2 = 1.0 / r2, rij = sqrt(r2), s = 1.0 / rij;
        double qq = qa * q[b], x = al * rij;
        double erfv = erf(x), derfc = NB_TWO_OVER_SQRTPI * exp(-x * x);
        double e2 = -qq * s * erfv;
        double df = qq * s * (s2 * erfv - s * al * derfc);
        gx += df * rx; gy += df * ry; gz += df * rz;
        ecorr += 0.5 * e2;
    }
    for (int k = p_off[a] + sub; act && k < p_off[a + 1]; k += EX_LANES) {
        int b = p_j[k];
        const double *p = p_par + 3 * (size_t)k;
        double rx = xa - coor[3 * (size_t)b], ry = ya - coor[3 * (size_t)b + 1], rz = za - coor[3 * (size_t)b + 2];
        double r2 = rx * rx + ry * ry + rz * rz, s2 = 1.0 / r2, e1 = 0, df1 = 0, e2 = 0, df2 = 0;
        if (p[0] > 1e-12) {
            double s6 = s2 * s2 * s2, A = p[0] * s6 * s6, B = p[1] * s6;
            e1 = A - B;
            df1 = -6.0 * s2 * (A + e1);
            vir14 -= 0.5 * df1 * r2;   // ener14_press.f:51-59
        }
        if (fabs(p[2]) > 1e-12) {
            double s = sqrt(s2);
            e2 = p[2] * s;
            df2 = -e2 * s2;
        }
        double df = df1 + df2;
        gx += df * rx; gy += df * ry; gz += df * rz;
        evdw14 += 0.5 * e1;
        eel14 += 0.5 * e2;
    }
    gx = sub_sum<EX_LANES>(gx); gy = sub_sum<EX_LANES>(gy); gz = sub_sum<EX_LANES>(gz);
    ecorr = sub_sum<EX_LANES>(ecorr); eel14 = sub_sum<EX_LANES>(eel14); evdw14 = sub_sum<EX_LANES>(evdw14);
    vir14 = sub_sum<EX_LANES>(vir14);
    if (!act || sub != 0) return;
    if (fixed_out) {   // mixed path: 2^32 fixed point, as the site gradients
        long long *gf = (long long *)grad + 3 * (size_t)a;
        gf[0] = __double2ll_rn(gx * NB_FIX_SCALE);
        gf[1] = __double2ll_rn(gy * NB_FIX_SCALE);
        gf[2] = __double2ll_rn(gz * NB_FIX_SCALE);
    } else {
        grad[3 * (size_t)a] = gx; grad[3 * (size_t)a + 1] = gy; grad[3 * (size_t)a + 2] = gz;
    }
    double *eo = e_out + NB_EX * (size_t)a;
    eo[0] = ecorr; eo[1] = eel14; eo[2] = evdw14; eo[3] = vir14;
}

// ---------------------------------------------------------------------------------
// End of an evaluation, one launch (k_finalize): gradient assembly in MOIL order, per-replica
// energies, and the status words and energies written to the host's page-locked copies by the
// blocks that have them.  Three launches and two copies took 22 us of a 216-water evaluation.

// Per-replica energies in two passes with a fixed partition, so large replicas spread over
// many blocks and the sums stay in a fixed order (deterministic):
//  energy_chunk: one block per chunk (EChunk: up to NB_FE_SEG consecutive units, atoms or PME
//    column items of one replica); every thread streams the chunk's flat array with a stride
//    that keeps its slot fixed (coalesced reads), the slots are summed by a halving tree;
//  energy_replica: the warp of the replica's last finished block adds its chunks' slot sums (a
//    lane per slot and chunk modulo four, then a fixed tree) and forms MOIL's energy names
//    (pot/eforce.f:122-204).
#define NB_FE_THREADS 256
static_assert(NB_FE_THREADS % NB_EU == 0 && NB_FE_THREADS % NB_EX == 0, "slot-preserving stride");
__device__ __forceinline__ void energy_chunk(int chunk, EChunk ch, const double *__restrict__ e_unit,
                                             const double *__restrict__ e_ex, const double *__restrict__ e_col,
                                             double *__restrict__ part)
{
    __shared__ double sh[NB_FE_THREADS];
    const int t = threadIdx.x;
    const int width = ch.kind <= 1 ? NB_EU : (ch.kind == 2 ? NB_EX : 1);
    const double *b = ch.kind <= 1 ? e_unit + (size_t)NB_EU * ch.begin
                                   : (ch.kind == 2 ? e_ex + (size_t)NB_EX * ch.begin : e_col + ch.begin);
    const int n = width * (ch.end - ch.begin);
    // four loads in flight per thread, four partial sums added in a fixed order
    double p[4] = {0.0, 0.0, 0.0, 0.0};
    int k = t;
    for (; k + 3 * NB_FE_THREADS < n; k += 4 * NB_FE_THREADS) {
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] += b[k + j * NB_FE_THREADS];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
        if (k + j * NB_FE_THREADS < n) p[j] += b[k + j * NB_FE_THREADS];
    sh[t] = (p[0] + p[1]) + (p[2] + p[3]);
    __syncthreads();
    // halving tree while the live range halves into a multiple of the slot width (thread k
    // adds k + half, which holds the same slot)
    int live = NB_FE_THREADS;
    while (live % 2 == 0 && (live / 2) % width == 0) {
        const int h = live / 2;
        if (t < h) sh[t] += sh[t + h];
        __syncthreads();
        live = h;
    }
    if (t < NB_EU) {
        double w = 0.0;
        if (t < width)
            for (int q = t; q < live; q += width) w += sh[q];
        part[(size_t)NB_EU * chunk + t] = w;
    }
}


__device__ __forceinline__ void energy_replica(int r, int lane, const RepDev *__restrict__ reps,
                                               const EChunk *__restrict__ chunks, const int *__restrict__ chunk_begin,
                                               const double *part, double *__restrict__ e_rep)
{
    const RepDev &R = reps[r];
    const int slot = lane % NB_EU;
    double a[4] = {0.0, 0.0, 0.0, 0.0};    // by chunk kind: this lane's slot over every fourth chunk
    const int c1 = chunk_begin[r + 1];
    for (int c = chunk_begin[r] + lane / NB_EU; c < c1; c += 32 / NB_EU) {
        const double v = __ldcg(part + (size_t)NB_EU * c + slot);
        const int kind = chunks[c].kind;
#pragma unroll
        for (int q = 0; q < 4; ++q) a[q] += kind == q ? v : 0.0;
    }
    double pw[NB_EU], po[NB_EU], px[NB_EX];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int o = NB_EU; o < 32; o <<= 1) a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
#pragma unroll
    for (int k = 0; k < NB_EU; ++k) {
        pw[k] = __shfl_sync(0xffffffffu, a[0], k);
        po[k] = __shfl_sync(0xffffffffu, a[1], k);
    }
#pragma unroll
    for (int k = 0; k < NB_EX; ++k) px[k] = __shfl_sync(0xffffffffu, a[2], k);
    const double cl = __shfl_sync(0xffffffffu, a[3], 0);
    if (lane != 0) return;
    const double elp = 0.5 * (pw[0] + po[0]), eli = 0.5 * (pw[1] + po[1]);
    const double eep = 0.5 * (pw[2] + po[2]), eei = 0.5 * (pw[3] + po[3]);
    const double npairs = 0.5 * (pw[4] + po[4]);
    // waters relative to the reference water (k_wref) add their reference energy here
    const double ecorr = px[0] + pw[5] + po[5] + (R.wref ? (double)R.nwat * R.wcorr0 : 0.0);
    const double eel14 = px[1], evdw14 = px[2];
    const double erec = 0.5 * cl;
    double *o = e_rep + NB_EREP * (size_t)r;
    o[0] = elp; o[1] = eep; o[2] = eli; o[3] = eei;          // e_vdw, e_el, e_vsym, e_lsym
    o[4] = eel14; o[5] = evdw14; o[6] = ecorr; o[7] = R.e_self; o[8] = erec;
    o[9] = elp + eep + eli + eei + eel14 + evdw14 + ecorr + R.e_self + erec;
    o[10] = eep + eei;
    o[11] = npairs;                                           // in-cutoff site pairs
    // LJ virial terms virvdw1..5 (MOIL's PRESS build): water-water primary and images,
    // other pairs primary and images, 1-4
    o[12] = 0.5 * pw[6]; o[13] = 0.5 * pw[7]; o[14] = 0.5 * po[6]; o[15] = 0.5 * po[7]; o[16] = px[3];
}

// the half-list kernel for a block size (128, 256 or 512 waters) and virial flag
using WaterHFn = decltype(&k_water_h<256, false>);
WaterHFn water_h_fn(int hb, bool vir)
{
    switch (hb) {
    case 128: return vir ? k_water_h<128, true> : k_water_h<128, false>;
    case 512: return vir ? k_water_h<512, true> : k_water_h<512, false>;
    default: return vir ? k_water_h<256, true> : k_water_h<256, false>;
    }
}

// Blocks [0, nchunk): energy chunks; the others: gradients of 256 atoms each.  st: status words
// (the kernels before this one are done with them), copied to the host's st_h and cleared
// for the next evaluation; a non-finite gradient sets *nan_h.  done: finished chunks per replica
// (zero between launches).  ctl: in an MD step, {evaluations since the last rebuild, -, sticky
// error bits}: the step's outcome goes there, and st[0] becomes the next step's rebuild request where
// the device decides on it (list_period > 0); list_period < 0: a step without a rebuild, whose lists a
// site has outrun (st[0]).
template <typename T>
__global__ void __launch_bounds__(NB_FE_THREADS) k_finalize(
    int nchunk, const EChunk *__restrict__ chunks, const int *__restrict__ chunk_begin,
    const double *__restrict__ e_unit, const double *__restrict__ e_ex, const double *__restrict__ e_col,
    double *__restrict__ epart, int *__restrict__ done, double *__restrict__ e_rep_h, int natom,
    const int *__restrict__ site_of, const int *__restrict__ atom_rep, const RepDev *__restrict__ reps,
    const long long *__restrict__ grad_site, const double *__restrict__ grad_ex, const T *__restrict__ part,
    const double *__restrict__ q, int nsw, const long long *__restrict__ fine, int nfine, double *__restrict__ dpot,
    int *__restrict__ st, int *__restrict__ st_h,
    int *__restrict__ nan_h, int *__restrict__ ctl, int list_period)
{
    const int t = threadIdx.x, b = blockIdx.x;
    if (b >= nchunk) {
        const int a = (b - nchunk) * NB_FE_THREADS + t;
        if (a >= natom) return;
        double g[3];
        if (!final_grad<T>(a, site_of, atom_rep, reps, grad_site, grad_ex, part, q, nsw, fine, nfine, g)) {
            *nan_h = 1;
            if (ctl) atomicOr(&ctl[2], NB_DEV_ERR_NAN);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) dpot[3 * (size_t)a + d] = g[d];
        return;
    }
    const EChunk ch = chunks[b];
    energy_chunk(b, ch, e_unit, e_ex, e_col, epart);
    if (t < 32) {
        // the chunk's sums are visible before it counts as finished
        __threadfence();
        __syncwarp();
        int last = 0;
        if (t == 0) last = atomicAdd(&done[ch.rep], 1) == chunk_begin[ch.rep + 1] - chunk_begin[ch.rep] - 1;
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) {
            __threadfence();
            energy_replica(ch.rep, t, reps, chunks, chunk_begin, epart, e_rep_h);
            if (t == 0) done[ch.rep] = 0;
        }
    }
    if (b == 0 && t == 0) {
        int s[8];
        for (int k = 0; k < 8; ++k) s[k] = st[k];
        for (int k = 0; k < 8; ++k) { st_h[k] = s[k]; st[k] = 0; }
        if (ctl) {
            if (s[0]) ctl[0] = 0;
            ctl[0] += 1;
            const int err = s[1] | (s[0] && list_period < 0 ? NB_DEV_STALE : 0);
            if (err) atomicOr(&ctl[2], err);
            // (no rebuild after an error)
            st[0] = list_period > 0 && ctl[0] >= list_period && (err | ctl[2]) == 0 ? 1 : 0;
        }
    }
}

// Lanes per water of the full-list kernel, from the waters of the whole handle (all replica
// groups, so a grouped handle gives the ungrouped one's bits): every lane of the GPU has work
// from a few thousand waters at 32 lanes each, and from then on fewer lanes lose less to
// partly filled rounds and to the sum over the lanes.  Water stage in us at 32 / 8 / 4 lanes:
// 1,334 waters 14 / 19 / 27, 3,000 22 / 19 / 28, 7,000 32 / 21 / 30, 12,000 46 / 34 / 32, 32,000
// 114 / 80 / 77, 110,860 (64 replicas) 366 / 197 / 175, 433,195 1418 / 733 / 633 (one water per
// thread: 78, 79, 82, 79, 120, 204, 657).  In a solute a water also has a long list of atoms (the
// solute system, 7,020 waters: 37 / 71 / 114; 34 at 32 lanes since its loop is packed; 5 of them, 35,100
// waters, a whole evaluation 337 / 299 / 290).
// 32-bit rows belong to replicas of 65,536 waters or more: four lanes.
int water_lanes(const NbCtx *c)
{
    if (!c->row16) return 4;
    return c->nw_handle <= (c->w2_handle < NB_W2_SOLUTE ? 4096 : 8192) ? 32 : (c->nw_handle <= 32768 ? 8 : 4);
}

using WaterSFn = decltype(&k_water_s<8, false, false, int>);
template <bool VIR, bool ATOMS>
WaterSFn water_s_fn(int lpw, bool row16)
{
    if (!row16) return k_water_s<4, VIR, ATOMS, int>;
    switch (lpw) {
    case 32: return k_water_s<32, VIR, ATOMS, unsigned short>;
    case 8: return k_water_s<8, VIR, ATOMS, unsigned short>;
    default: return k_water_s<4, VIR, ATOMS, unsigned short>;
    }
}
// (atoms: of the whole handle, so every replica group runs the same kernel)
WaterSFn water_s_fn(int lpw, bool vir, bool atoms, bool row16)
{
    if (atoms) return vir ? water_s_fn<true, true>(lpw, row16) : water_s_fn<false, true>(lpw, row16);
    return vir ? water_s_fn<true, false>(lpw, row16) : water_s_fn<false, false>(lpw, row16);
}

template <typename T>
void water_t(NbCtx *c)
{
    cudaStream_t s = c->stream;
    if (c->timing) cudaEventRecord(c->ev[2], s);
    if (sizeof(T) == 4 && c->nW > 0 && c->whalf) {
        water_h_fn(c->hb, c->virial)<<<(int)c->hblocks.size(), c->hb, (size_t)36 * c->jsh, s>>>(
            c->d_hblocks, c->d_reps, (const float4 *)c->d_pos, (const float4 *)c->d_woff, c->d_site_lj,
            c->d_site_flags, c->d_hrow, c->caph, c->d_hcnt, c->d_jset, c->d_jn, c->jcap, c->jsh, c->d_wl2_off, c->d_wl2,
            cap_int(c->cap_wl2), c->d_grad_site, c->d_e_unit, c->water_excl_fast);
        c->launches++;
    } else if (c->nW > 0) {
        if constexpr (sizeof(T) == 4) {
            const int lpw = water_lanes(c);
            water_s_fn(lpw, c->virial, c->na_handle > 0, c->row16)<<<(int)((c->nW * lpw + WBLOCK - 1) / WBLOCK), WBLOCK, 0, s>>>(
                (int)c->nW, c->d_reps, c->d_site_rep, (const float4 *)c->d_pos, (const float4 *)c->d_woff,
                c->d_site_lj, c->d_site_flags, c->d_wl1_cnt, c->d_wl1, c->cap_row1, c->d_wl2_off, c->d_wl2,
                cap_int(c->cap_wl2), c->d_grad_site, c->d_e_unit, c->water_excl_fast);
        } else {
            (c->row16 ? k_water_d<unsigned short> : k_water_d<int>)<<<(int)((c->nW + WARPS64 - 1) / WARPS64),
                                                                      32 * WARPS64, 0, s>>>(
                (int)c->nW, c->d_reps, c->d_site_rep, (const double4 *)c->d_pos, (const double4 *)c->d_woff,
                c->d_site_lj, c->d_site_flags, c->d_wl1_cnt, c->d_wl1, c->cap_row1, c->d_wl2_off, c->d_wl2,
                cap_int(c->cap_wl2), (unsigned long long *)c->d_grad_site, (unsigned long long *)c->d_grad_fine,
                c->d_e_unit);
        }
        c->launches++;
    }
    if (c->timing) cudaEventRecord(c->ev[3], s);
}

}  // namespace

void nb_launch_water(NbCtx *c)
{
    // the kernels that evaluate each water pair once add both sides with atomics: the water
    // sites' gradient starts at zero
    if (c->nW > 0 && (c->precision == MOIL_NB_FP64 || c->whalf))
        cudaMemsetAsync(c->d_grad_fine ? c->d_grad_fine : c->d_grad_site, 0,
                        sizeof(long long) * (c->d_grad_fine ? 18 : 9) * (size_t)c->nW, c->stream);
    if (c->precision == MOIL_NB_FP64) water_t<double>(c);
    else water_t<float>(c);
}

void nb_launch_atoms(NbCtx *c)
{
    cudaStream_t s = c->stream;
    if (c->nA > 0) {
        const int nb = (int)((c->nA + 3) / 4);
        if (c->precision == MOIL_NB_FP64)
            k_atom_d<<<nb, 128, 0, s>>>((int)c->nA, (int)c->nW, c->d_reps, c->d_site_rep, c->d_pos, c->d_site_lj,
                                        c->d_site_flags, c->d_xl_off, c->d_xl, cap_int(c->cap_xl), c->d_grad_site,
                                        c->d_e_unit);
        else
            k_atom_f<<<nb, 128, 0, s>>>((int)c->nA, (int)c->nW, c->d_reps, c->d_site_rep, (const float4 *)c->d_pos,
                                        (const float2 *)c->d_site_lj, c->d_site_flags, c->d_xl_off, c->d_xl,
                                        cap_int(c->cap_xl), c->d_grad_site, c->d_e_unit);
        c->launches++;
    }
    if (c->timing) cudaEventRecord(c->ev[4], s);
}

// shared-memory carveout (percent of the per-SM maximum) for `bytes` of resident blocks
static int carveout_pct(NbCtx *c, size_t bytes)
{
    int smax = 0;
    if (cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c->device) != cudaSuccess || smax <= 0)
        return 100;
    return (int)std::min<size_t>(100, (100 * bytes + smax - 1) / smax);
}

int nb_realspace_configure(NbCtx *c)
{
    // full-list FP32 water kernels: four resident blocks of static shared memory; the smallest
    // carveout that holds them leaves the most L1 for the partner-record gathers
    for (int lpw : {32, 8, 4})
        for (int k = 0; k < 8; ++k) {
            const void *fn = (const void *)water_s_fn(lpw, k & 1, k & 2, k & 4);
            cudaFuncAttributes fa;
            NB_CUDA_OK(c, cudaFuncGetAttributes(&fa, fn));
            NB_CUDA_OK(c, cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                               carveout_pct(c, 4 * (fa.sharedSizeBytes + 1024))));
        }
    return MOIL_NB_OK;
}

// the half-list kernel keeps two resident blocks per SM (its register budget) with the
// current j-set capacity
bool nb_half_two_blocks(NbCtx *c)
{
    int smax = 0;
    cudaFuncAttributes fa;
    const void *fn = (const void *)water_h_fn(c->hb, false);
    if (cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c->device) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, fn) != cudaSuccess)
        return false;
    const int per_sm = 512 / c->hb;
    return (size_t)per_sm * ((size_t)36 * c->jcap + fa.sharedSizeBytes + 1024) <= (size_t)smax;
}

int nb_half_configure(NbCtx *c)
{
    int optin = 0;
    NB_CUDA_OK(c, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
    const void *fns[2] = {(const void *)water_h_fn(c->hb, false), (const void *)water_h_fn(c->hb, true)};
    // Accumulators in shared memory: 9.5 per water of the block.  The blocks of an SM then take 175 KB; the
    // next carveout leaves too little L1 for the partner records (256 waters a block, 512 replicas,
    // evaluation in us: 2,430 partners 2179, 2,560 2453, 1,560 2196), and the few partners beyond go
    // straight to the gradient (32,000 waters: 2,230 and 2,430 167, 1,780 212).
    c->jsh = nb_half_two_blocks(c) ? std::min(c->jcap, 19 * c->hb / 2) : c->jcap;
    const size_t dyn = (size_t)36 * c->jsh;
    for (const void *fn : fns) {
        cudaFuncAttributes fa;
        NB_CUDA_OK(c, cudaFuncGetAttributes(&fa, fn));
        if (c->jcap > 65535 || (size_t)36 * c->jcap + fa.sharedSizeBytes > (size_t)optin) return MOIL_NB_ERR_OVERFLOW;
        // the limit belongs to the kernel, not to the handle: other handles (replica groups)
        // may launch it with larger j-sets, so it only ever grows
        if ((int)dyn > fa.maxDynamicSharedSizeBytes)
            NB_CUDA_OK(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
        // the smallest shared-memory carveout that holds the resident blocks (512 / hb per SM):
        // the rest of the SM's unified memory stays L1 for the partner-record gathers
        NB_CUDA_OK(c, cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                           carveout_pct(c, (512 / c->hb) * (dyn + fa.sharedSizeBytes))));
    }
    return MOIL_NB_OK;
}

void nb_launch_excl14(NbCtx *c, const double *d_coor)
{
    const int fast = c->water_excl_fast && c->nW > 0;
    // mixed path: the water kernels add each water's own corrections
    if (fast && c->precision == MOIL_NB_FP64) {
        k_excl_water<<<(int)((c->nW + 31) / 32), 32, 0, c->stream>>>(
            (int)c->nW, c->d_unit_atom, c->d_atom_rep, c->d_reps, d_coor, c->d_q, c->d_grad_ex, c->d_e_ex);
        c->launches++;
    }
    if (!fast || c->nA > 0) {
        // the atoms outside waters (the units after the waters), or all of them
        const int64_t n = fast ? c->nA : c->natom;
        k_excl14<<<(int)((n * EX_LANES + 31) / 32), 32, 0, c->stream>>>(
            (int)n, fast ? c->d_unit_atom + c->nW : nullptr, c->d_atom_rep, c->d_reps, d_coor, c->d_q, c->d_ex_off,
            c->d_ex_j, c->d_p14_off, c->d_p14_j, c->d_p14_par, c->precision != MOIL_NB_FP64, c->d_grad_ex, c->d_e_ex);
        c->launches++;
    }
}

void nb_launch_finalize(NbCtx *c, double *d_dpot, int *ctl, EvalMode mode)
{
    const int period = mode == EVAL_DEVICE ? c->list_period : (mode == EVAL_KEEP ? -1 : 0);
    // (no gradient where the integrator forms it itself)
    const int nchunk = (int)c->echunks.size(),
              nb = nchunk + (d_dpot ? (int)((c->natom + NB_FE_THREADS - 1) / NB_FE_THREADS) : 0);
    auto launch = [&](auto kernel, auto part, int nsw) {
        kernel<<<nb, NB_FE_THREADS, 0, c->stream>>>(
            nchunk, c->d_echunks, c->d_echunk_begin, c->d_e_unit, c->d_e_ex, c->d_e_col, c->d_epart, c->d_edone,
            c->h_e_rep, (int)c->natom, c->d_site_of, c->d_atom_rep, c->d_reps, c->d_grad_site, c->d_grad_ex, part,
            c->d_q, nsw, c->d_grad_fine, c->d_grad_fine ? (int)(3 * c->nW) : 0, d_dpot, c->d_status, c->h_status, c->h_status + 23, ctl, period);
    };
    if (c->precision == MOIL_NB_FP64) launch(k_finalize<double>, (const double *)c->d_part, 0);
    else launch(k_finalize<float>, (const float *)c->d_part, c->water_excl_fast ? (int)(3 * c->nW) : 0);
    c->launches++;
}
