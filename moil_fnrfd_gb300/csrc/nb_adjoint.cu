// nb_adjoint.cu -- parameter derivatives of the nonbonded energy: dE/dq, dE/deps and
// dE/dsigma per atom (moil_nb_adjoint).  MOIL computes none of them; the oracle's
// ora_adjoint_mi is the reference, itself checked against finite differences.
//
// One evaluation (moil_nb_eval semantics) leaves the lists, the site-ordered positions and
// the PME grid on the device (the real potential planes on the mixed path, the convolved
// spectrum on the plain path, whose inverse plane kernel then gives each site's potential
// shares); these kernels then accumulate (FP64; mixed path: pair sums and the grid's part as hi + lo FP32
// pairs):
//   dE/dq_i     = sum over i's real-space partners of k q_j erfc(alpha r)/r
//               - sum over i's excluded partners of k q_j erf(alpha r)/r
//               + 1-4 Coulomb p14(3)/(q_i r) + fc * sum(theta * potential grid)
//               - 2 alpha/sqrt(pi) k q_i                      (k = kofdie/eps, fc = sqrt(k))
//   dE/deps_i   = sum over i's LJ pairs of (A - B) / (2 eps_i)     (A ~ r^-12, B ~ r^-6 parts)
//   dE/dsigma_i = sum over i's LJ pairs of (6A - 3B) / sigma_i   (geometric: sigma_ij^6 =
//                 sigma_i^3 sigma_j^3), or / sigma_ij with sigma_ij = (sigma_i + sigma_j)/2
//                 (arithmetic)
// with eps and sigma decoded from MOIL's epsgm encoding (connect/fillpt.f:136-184).  The
// pair predicates are the energy kernels' (MOIL's, pot/watwat_ewald.f, pot/cdie_ewald.f);
// water-water Coulomb uses each site's own charge (MOIL's water kernel the last water's,
// the same for identical waters).  The LJ switch extension is not differentiated.
#include "nb_internal.h"
#include "nb_pair.cuh"

namespace {

// geometric: epsgm12 = 2 sqrt(eps) sigma^6, epsgm6 = 2 sqrt(eps) sigma^3;
// arithmetic: epsgm12 = 2 sqrt(eps), epsgm6 = sigma
__device__ __forceinline__ void lj_decode(int arith, double e12, double e6, double &eps, double &sig)
{
    if (arith) {
        eps = 0.25 * e12 * e12;
        sig = e6;
    } else if (e12 > 0.0 && e6 > 0.0) {
        const double se = e6 * e6 / (2.0 * e12);
        sig = cbrt(e12 / e6);
        eps = se * se;
    } else {
        eps = 0.0;
        sig = 0.0;
    }
}

// the pair's LJ energy parts a (r^-12) and b (r^-6) into atom i's derivatives
__device__ __forceinline__ void lj_adj(int arith, double a, double b, double eps_i, double sig_i, double sig_j,
                                       double &de, double &ds)
{
    const double e = a - b, g = 6.0 * a - 3.0 * b;
    if (eps_i > 0.0) de += e / (2.0 * eps_i);
    if (!arith) {
        if (sig_i > 0.0) ds += g / sig_i;
    } else {
        const double sij = 0.5 * (sig_i + sig_j);
        if (sij > 0.0) ds += g / sij;
    }
}

// LJ parts of a non-water pair (cdie_ewald.f:377-383 geometric, :432-472 arithmetic)
__device__ __forceinline__ void lj_parts(int arith, double e12i, double e6i, double e12j, double e6j, double s2,
                                         double &a, double &b)
{
    const double s6 = s2 * s2 * s2;
    if (!arith) {
        a = e12i * e12j * s6 * s6;
        b = e6i * e6j * s6;
    } else {
        const double aa = e12i * e12j, sg = 0.5 * (e6i + e6j);
        double b1 = sg * sg * sg;
        b1 = b1 * b1;
        b = aa * b1 * s6;
        a = aa * b1 * b1 * s6 * s6;
    }
}

// Plain FP64 path
// one non-water-semantics site pair (atom_pair of the energy kernels) into site i's sums
__device__ __forceinline__ void atom_pair_adj(const RepDev &R, double r2, double qi, double qj, double2 lji,
                                              double2 ljj, unsigned fi, unsigned fj, double &phi, double &de,
                                              double &ds)
{
    const bool hr = !R.arith && R.hvdw0 && ((fi | fj) & SF_HTINY) && r2 < (double)R.re2;
    const bool lj = r2 < (double)R.rv2 && !hr;
    const bool el = r2 < (double)R.rmax2 && qi * qj != 0.0;
    if (el) {
        const double r = sqrt(r2);
        phi += R.epstmp * qj * erfc(R.alphad * r) / r;
    }
    if (lj) {
        double a, b, ei, si, ej, sj;
        lj_parts(R.arith, lji.x, lji.y, ljj.x, ljj.y, 1.0 / r2, a, b);
        lj_decode(R.arith, lji.x, lji.y, ei, si);
        lj_decode(R.arith, ljj.x, ljj.y, ej, sj);
        lj_adj(R.arith, a, b, ei, si, sj, de, ds);
    }
}

// one warp per water: W1 (nine site pairs per molecule pair) and W2, the lanes taking the
// entries of both lists in turn
template <typename E>
__global__ void __launch_bounds__(128) k_adj_water(int nW, const RepDev *__restrict__ reps, const int *__restrict__ site_rep,
                            const int *__restrict__ site_orig, const double4 *__restrict__ pos,
                            const double4 *__restrict__ woff, const double2 *__restrict__ lj,
                            const unsigned *__restrict__ sflags, const int2 *__restrict__ wl1_cnt,
                            const void *__restrict__ wl1, int cap_row, const int *__restrict__ wl2_off,
                            const int *__restrict__ wl2, int cap2, double *__restrict__ dq, double *__restrict__ de,
                            double *__restrict__ ds)
{
    const int lane = threadIdx.x & 31, i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= nW) return;
    const RepDev &R = reps[site_rep[3 * i]];
    const double4 oi = pos[3 * i];
    const double4 h1 = woff[3 * i + 1], h2 = woff[3 * i + 2];
    const double hi[3][3] = {{0.0, 0.0, 0.0}, {h1.x, h1.y, h1.z}, {h2.x, h2.y, h2.z}};
    double phi[3] = {0, 0, 0}, dE[3] = {0, 0, 0}, dS[3] = {0, 0, 0};
    double epsO, sigO;
    const double2 ljO = lj[3 * i];
    lj_decode(R.arith, ljO.x, ljO.y, epsO, sigO);
    const int2 c = wl1_cnt[i];
    const int nn = min(c.x, cap_row), n = min(c.x + c.y, cap_row);
    const E *row = (const E *)wl1 + (size_t)i * cap_row;
    const int base = sizeof(E) == 2 ? R.wat0 : 0;   // uint16 entries: offsets from the replica's first water
    for (int v = lane; v < n; v += 32) {
        const int j = base + (int)row[v < nn ? v : cap_row - 1 - (v - nn)];
        const double4 oj = pos[3 * j];
        double dx = oi.x - oj.x, dy = oi.y - oj.y, dz = oi.z - oj.z;
        const double nx = nb_rint(dx * R.invLd[0]), ny = nb_rint(dy * R.invLd[1]), nz = nb_rint(dz * R.invLd[2]);
        dx = nb_shift(R, 0, dx, nx);
        dy = nb_shift(R, 1, dy, ny);
        dz = nb_shift(R, 2, dz, nz);
        const double r2oo = dx * dx + dy * dy + dz * dz;
        if (r2oo > (double)R.rmax2) continue;
        const double4 j1 = woff[3 * j + 1], j2 = woff[3 * j + 2];
        const double hj[3][3] = {{0.0, 0.0, 0.0}, {j1.x, j1.y, j1.z}, {j2.x, j2.y, j2.z}};
        const double qj[3] = {oj.w, pos[3 * j + 1].w, pos[3 * j + 2].w};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const double ex = hi[a][0] + dx - hj[b][0], ey = hi[a][1] + dy - hj[b][1],
                             ez = hi[a][2] + dz - hj[b][2];
                const double r = sqrt(ex * ex + ey * ey + ez * ez);
                phi[a] += R.epstmp * qj[b] * erfc(R.alphad * r) / r;
            }
        if (r2oo <= (double)R.rv2) {
            const double s2 = 1.0 / r2oo, s6 = s2 * s2 * s2;
            double ej, sj;
            const double2 ljj = lj[3 * j];
            lj_decode(R.arith, ljj.x, ljj.y, ej, sj);
            lj_adj(R.arith, R.w12d * s6 * s6, R.w6d * s6, epsO, sigO, sj, dE[0], dS[0]);
        }
    }
    for (int k = min(wl2_off[i], cap2) + lane; k < min(wl2_off[i + 1], cap2); k += 32) {
        const int s = wl2[k];
        const double4 xj = pos[s];
        const double2 ljj = lj[s];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double4 xi = pos[3 * i + a];
            double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            dx = nb_shift(R, 0, dx, nb_rint(dx * R.invLd[0]));
            dy = nb_shift(R, 1, dy, nb_rint(dy * R.invLd[1]));
            dz = nb_shift(R, 2, dz, nb_rint(dz * R.invLd[2]));
            atom_pair_adj(R, dx * dx + dy * dy + dz * dz, xi.w, xj.w,
                             lj[3 * i + a], ljj, sflags[3 * i + a], sflags[s], phi[a], dE[a], dS[a]);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        phi[a] = sub_sum<32>(phi[a]); dE[a] = sub_sum<32>(dE[a]); dS[a] = sub_sum<32>(dS[a]);
        if (lane != a) continue;
        const int o = site_orig[3 * i + a];
        dq[o] = phi[a];
        de[o] = dE[a];
        ds[o] = dS[a];
    }
}

// one warp per non-water atom over its X list
__global__ void __launch_bounds__(128) k_adj_atom(int nA, int nW, const RepDev *__restrict__ reps, const int *__restrict__ site_rep,
                           const int *__restrict__ site_orig, const double4 *__restrict__ pos, const double2 *__restrict__ lj,
                           const unsigned *__restrict__ sflags, const int *__restrict__ xl_off,
                           const int *__restrict__ xl, int capx, double *__restrict__ dq, double *__restrict__ de,
                           double *__restrict__ ds)
{
    const int lane = threadIdx.x & 31, k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= nA) return;
    const int si = 3 * nW + k;
    const RepDev &R = reps[site_rep[si]];
    const double4 xi = pos[si];
    const double2 lji = lj[si];
    double phi = 0, dE = 0, dS = 0;
    for (int q = min(xl_off[k], capx) + lane; q < min(xl_off[k + 1], capx); q += 32) {
        const int s = xl[q];
        const double4 xj = pos[s];
        double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        dx = nb_shift(R, 0, dx, nb_rint(dx * R.invLd[0]));
        dy = nb_shift(R, 1, dy, nb_rint(dy * R.invLd[1]));
        dz = nb_shift(R, 2, dz, nb_rint(dz * R.invLd[2]));
        atom_pair_adj(R, dx * dx + dy * dy + dz * dz, xi.w, xj.w, lji,
                         lj[s], sflags[si], sflags[s], phi, dE, dS);
    }
    phi = sub_sum<32>(phi); dE = sub_sum<32>(dE); dS = sub_sum<32>(dS);
    if (lane != 0) return;
    const int o = site_orig[si];
    dq[o] = phi;
    de[o] = dE;
    ds[o] = dS;
}

// ---------------------------------------------------------------------------------
// Mixed path: the same sums with FP32 pair arithmetic (the energy kernels' erfc fit and a
// Newton-refined reciprocal square root), summed per site in FP32 over chunks of CHUNK_ADJ list
// entries and then as hi + lo pairs -- the FP64 pipe of this GPU is 1/64 of the FP32 one: per-pair
// FP64 erfc, square roots and divisions would dominate, and even FP64 sums over the lanes at a
// list's end took a quarter of the water kernel.  k = kofdie/eps is applied to the potential sums at
// the end.
#define CHUNK_ADJ 64

// 1/sqrt(r2) to about an ulp: the approximate MUFU value and one Newton step
__device__ __forceinline__ float adj_rsqrt(float r2)
{
    const float y = nb_rsqrt_approx(r2);
    return fmaf(-0.5f * y, fmaf(r2, y * y, -1.f), y);
}

// erfc(alpha r) / r (the erfc fit of ewald1)
__device__ __forceinline__ float adj_pot(const WaterK &K, float r2, float rinv)
{
    const float tt = nb_rcp_approx(fmaf(K.palpha, r2 * rinv, 1.f)), u = fmaf(ERFCX_A, tt, ERFCX_B);
    const float C[ERFCX_NC] = ERFCX_COEFS;
    float p = C[ERFCX_NC - 1];
#pragma unroll
    for (int m = ERFCX_NC - 2; m >= 0; --m) p = fmaf(p, u, C[m]);
    return nb_ex2_approx(-r2 * K.ex2c) * (tt * p) * rinv;
}
__device__ __forceinline__ float2 adj_pot2(const WaterK &K, float2 r2)
{
    const float2 y = f2(nb_rsqrt_approx(r2.x), nb_rsqrt_approx(r2.y));
    const float2 rinv = __ffma2_rn(__fmul2_rn(f2(-0.5f), y), __ffma2_rn(r2, __fmul2_rn(y, y), f2(-1.f)), y);
    const float2 den = __ffma2_rn(f2(K.palpha), __fmul2_rn(r2, rinv), f2(1.f)), arg = __fmul2_rn(r2, f2(K.ex2c));
    const float2 tt = f2(nb_rcp_approx(den.x), nb_rcp_approx(den.y)), u = __ffma2_rn(f2(ERFCX_A), tt, f2(ERFCX_B));
    const float C[ERFCX_NC] = ERFCX_COEFS;
    float2 p = f2(C[ERFCX_NC - 1]);
#pragma unroll
    for (int m = ERFCX_NC - 2; m >= 0; --m) p = __ffma2_rn(p, u, f2(C[m]));
    return __fmul2_rn(__fmul2_rn(f2(nb_ex2_approx(-arg.x), nb_ex2_approx(-arg.y)), __fmul2_rn(tt, p)), rinv);
}

// eps and sigma from the epsgm encoding in FP32 (as lj_decode)
__device__ __forceinline__ void lj_decode_f(int arith, float e12, float e6, float &eps, float &sig)
{
    if (arith) {
        eps = 0.25f * e12 * e12;
        sig = e6;
    } else if (e12 > 0.f && e6 > 0.f) {
        const float se = e6 * e6 / (2.f * e12);
        sig = cbrtf(e12 / e6);
        eps = se * se;
    } else {
        eps = 0.f;
        sig = 0.f;
    }
}

// a site's own factors of the LJ derivatives: 1/(2 eps), sigma and 1/sigma (0 where there is none)
struct AdjLJ {
    float2 lj;
    float inv2e, sig, isig;
    __device__ AdjLJ(int arith, float2 v) : lj(v)
    {
        float e;
        lj_decode_f(arith, v.x, v.y, e, sig);
        inv2e = e > 0.f ? 0.5f / e : 0.f;
        isig = sig > 0.f ? 1.f / sig : 0.f;
    }
};

// LJ parts of a non-water pair into site i's derivatives
__device__ __forceinline__ void adj_lj(const AtomK &A, float rinv, const AdjLJ &i, float2 ljj, float &de, float &ds)
{
    const float s2 = rinv * rinv, s6 = s2 * s2 * s2;
    float a, b, is;
    if (!A.arith) {
        a = i.lj.x * ljj.x * s6 * s6;
        b = i.lj.y * ljj.y * s6;
        is = i.isig;
    } else {
        const float sij = 0.5f * (i.lj.y + ljj.y);
        float b1 = sij * sij * sij;
        b1 = b1 * b1;
        b = i.lj.x * ljj.x * b1 * s6;
        a = b * b1 * s6;
        const float y = nb_rcp_approx(sij);            // refined to about an ulp
        is = sij > 0.f ? fmaf(y, fmaf(-sij, y, 1.f), y) : 0.f;
    }
    de = fmaf(a - b, i.inv2e, de);
    ds = fmaf(6.f * a - 3.f * b, is, ds);
}

// one non-water-semantics site pair (atom_pair of the energy kernels): q_j erfc(alpha r)/r into
// phi (k applied later), the LJ parts into de, ds of site i
__device__ __forceinline__ void atom_pair_adj_f(const AtomK &A, float r2, bool qi, float qj, const AdjLJ &i, float2 ljj,
                                                bool tiny, float &phi, float &de, float &ds)
{
    const bool lj = r2 < A.rv2 && !(tiny && r2 < A.re2), el = r2 < A.rmax2 && qi && qj != 0.f;
    if (!el && !lj) return;
    const float rinv = adj_rsqrt(r2);
    if (el) phi = fmaf(qj, adj_pot(A.K, r2, rinv), phi);
    if (lj) adj_lj(A, rinv, i, ljj, de, ds);
}

// LPW lanes per water (FP32 pairs): W1 (nine site pairs per molecule pair, eight of them packed two
// by two, and the O-O LJ) and W2 (the H sites packed), the lanes taking the entries of both lists
// in turn, partner records one entry ahead.  Bound: FP32 issue.  One water per thread: 249 us for
// the 460 waters of a small solute system.  8 systems of 7,020 waters and 2,496 atoms: scalar pairs
// and FP64 sums 193 us, this 114.
template <int LPW, typename E>
__global__ void __launch_bounds__(128) k_adj_water_f(int nW, const RepDev *__restrict__ reps,
                                                     const int *__restrict__ site_rep,
                                                     const int *__restrict__ site_orig,
                                                     const float4 *__restrict__ pos, const float4 *__restrict__ woff,
                                                     const float2 *__restrict__ lj,
                                                     const unsigned *__restrict__ sflags,
                                                     const int2 *__restrict__ wl1_cnt, const void *__restrict__ wl1,
                                                     int cap_row, const int *__restrict__ wl2_off,
                                                     const int *__restrict__ wl2, int cap2, double *__restrict__ dq,
                                                     double *__restrict__ de, double *__restrict__ ds)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, sub = t & (LPW - 1);
    const bool act = t / LPW < nW;
    const int i = act ? t / LPW : nW - 1;    // idle lanes of the last block: empty lists, no output
    const RepDev &R = reps[site_rep[3 * i]];
    const AtomK A(R);
    const float w12 = R.w12, w6 = R.w6;
    const float4 oi = woff[3 * i], h1 = woff[3 * i + 1], h2 = woff[3 * i + 2];
    const float2 hx = f2(h1.x, h2.x), hy = f2(h1.y, h2.y), hz = f2(h1.z, h2.z);
    float2 phi[3], dE[3], dS[3];             // sums of chunks, hi + lo
#pragma unroll
    for (int a = 0; a < 3; ++a) { phi[a] = f2(0.f); dE[a] = f2(0.f); dS[a] = f2(0.f); }
    float p0 = 0.f, e3[3] = {0.f, 0.f, 0.f}, s3[3] = {0.f, 0.f, 0.f};
    float2 pO = f2(0.f), pH = f2(0.f);       // potential at O from (H1, H2), at (H1, H2)
    auto flush = [&]() {
        two_add(phi[0], p0 + (pO.x + pO.y)); two_add(phi[1], pH.x); two_add(phi[2], pH.y);
        p0 = 0.f; pO = f2(0.f); pH = f2(0.f);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            two_add(dE[a], e3[a]); two_add(dS[a], s3[a]);
            e3[a] = 0.f; s3[a] = 0.f;
        }
    };
    const AdjLJ lO(R.arith, lj[3 * i]);
    auto pair = [&](float4 oj, float4 j1, float4 j2) {
        float dx = oi.x - oj.x, dy = oi.y - oj.y, dz = oi.z - oj.z;
        bool img;
        A.image(dx, dy, dz, img);
        const float r2oo = dx * dx + dy * dy + dz * dz;
        if (r2oo <= A.rmax2) {
            const float ri = adj_rsqrt(r2oo);
            p0 = fmaf(oj.w, adj_pot(A.K, r2oo, ri), p0);
            if (r2oo <= A.rv2) {
                const float s2 = ri * ri, s6 = s2 * s2 * s2, a = w12 * s6 * s6, b = w6 * s6;
                e3[0] = fmaf(a - b, lO.inv2e, e3[0]);
                s3[0] = fmaf(6.f * a - 3.f * b, lO.isig, s3[0]);  // sigma_ij = sigma_O for water pairs (both rules)
            }
            {
                // O of i with (H1, H2) of j
                const float2 x = f2(dx - j1.x, dx - j2.x), y = f2(dy - j1.y, dy - j2.y), z = f2(dz - j1.z, dz - j2.z);
                pO = __ffma2_rn(f2(j1.w, j2.w), adj_pot2(A.K, __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z)))), pO);
            }
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                // (H1, H2) of i with site s of j
                const float qx = s == 0 ? dx : (s == 1 ? dx - j1.x : dx - j2.x);
                const float qy = s == 0 ? dy : (s == 1 ? dy - j1.y : dy - j2.y);
                const float qz = s == 0 ? dz : (s == 1 ? dz - j1.z : dz - j2.z);
                const float2 x = __fadd2_rn(hx, f2(qx)), y = __fadd2_rn(hy, f2(qy)), z = __fadd2_rn(hz, f2(qz));
                pH = __ffma2_rn(f2(s == 0 ? oj.w : (s == 1 ? j1.w : j2.w)),
                                adj_pot2(A.K, __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z)))), pH);
            }
        }
    };
    const W1Row<E> row(wl1_cnt, wl1, cap_row, i, R.wat0);
    const int n = act ? row.n : 0;
    int cnt = 0;
    if (sub < n) {
        // two record buffers in turn, as in k_water_s
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
            if (cnt >= CHUNK_ADJ) { flush(); cnt = 0; }
        }
    }
    __syncwarp();     // rows differ in length: the lanes that end early wait here
    const int q0 = min(wl2_off[i], cap2), q1 = act ? min(wl2_off[i + 1], cap2) : q0;
    if (q0 + sub < q1) {
        const float4 xo = pos[3 * i], x1 = pos[3 * i + 1], x2 = pos[3 * i + 2];
        const AdjLJ l1(R.arith, lj[3 * i + 1]), l2(R.arith, lj[3 * i + 2]);
        const bool to = A.tiny && (sflags[3 * i] & SF_HTINY), t1 = A.tiny && (sflags[3 * i + 1] & SF_HTINY),
                   t2 = A.tiny && (sflags[3 * i + 2] & SF_HTINY);
        auto entry = [&](int k) { return wl2[min(k, q1 - 1)]; };
        int sb = entry(q0 + sub), sn = entry(q0 + sub + LPW);
        float4 xb = pos[sb];
        float2 lb = lj[sb];
        for (int k = q0 + sub; k < q1; k += LPW) {
            const int s = sb;
            const float4 xj = xb;
            const float2 ljj = lb;
            sb = sn;
            xb = pos[sb]; lb = lj[sb];
            sn = entry(k + 2 * LPW);
            const bool tj = A.tiny && (sflags[s] & SF_HTINY);
            float dx = xo.x - xj.x, dy = xo.y - xj.y, dz = xo.z - xj.z;
            bool img;
            A.image(dx, dy, dz, img);
            atom_pair_adj_f(A, dx * dx + dy * dy + dz * dz, xo.w != 0.f, xj.w, lO, ljj, to || tj, p0, e3[0], s3[0]);
            float2 x = f2(x1.x - xj.x, x2.x - xj.x), y = f2(x1.y - xj.y, x2.y - xj.y), z = f2(x1.z - xj.z, x2.z - xj.z);
            float2 nx, ny, nz;
            A.image2(x, y, z, nx, ny, nz);
            const float2 r2 = __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z)));
            const bool i1 = r2.x < A.rmax2 && x1.w * xj.w != 0.f, i2 = r2.y < A.rmax2 && x2.w * xj.w != 0.f;
            if (i1 || i2) {
                const float2 f = adj_pot2(A.K, r2);
                pH = __ffma2_rn(f2(i1 ? f.x : 0.f, i2 ? f.y : 0.f), f2(xj.w), pH);
            }
            if (l1.inv2e != 0.f) {
                if (r2.x < A.rv2 && !((t1 || tj) && r2.x < A.re2)) adj_lj(A, adj_rsqrt(r2.x), l1, ljj, e3[1], s3[1]);
            }
            if (l2.inv2e != 0.f) {
                if (r2.y < A.rv2 && !((t2 || tj) && r2.y < A.re2)) adj_lj(A, adj_rsqrt(r2.y), l2, ljj, e3[2], s3[2]);
            }
            if (++cnt >= CHUNK_ADJ) { flush(); cnt = 0; }
        }
    }
    __syncwarp();
    flush();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float2 f = sub_two_sum<LPW>(phi[a]), e = sub_two_sum<LPW>(dE[a]), s = sub_two_sum<LPW>(dS[a]);
        if (!act || sub != a) continue;
        const int o = site_orig[3 * i + a];
        dq[o] = R.epstmp * ((double)f.x + (double)f.y);
        de[o] = (double)e.x + (double)e.y;
        ds[o] = (double)s.x + (double)s.y;
    }
}

// one warp per non-water atom over its X list (FP32 pairs), records one entry ahead; one atom per
// thread: 434 us for 209 atoms.  19,968 atoms: 136 us with FP64 sums and the constants loaded again
// for every pair, this 49.
__global__ void __launch_bounds__(128) k_adj_atom_f(int nA, int nW, const RepDev *__restrict__ reps,
                                                    const int *__restrict__ site_rep,
                                                    const int *__restrict__ site_orig, const float4 *__restrict__ pos,
                                                    const float2 *__restrict__ lj, const unsigned *__restrict__ sflags,
                                                    const int *__restrict__ xl_off, const int *__restrict__ xl, int capx,
                                                    double *__restrict__ dq, double *__restrict__ de,
                                                    double *__restrict__ ds)
{
    const int lane = threadIdx.x & 31, k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= nA) return;
    const int si = 3 * nW + k;
    const RepDev &R = reps[site_rep[si]];
    const AtomK A(R);
    const float4 xi = pos[si];
    const AdjLJ li(R.arith, lj[si]);
    const bool ti = A.tiny && (sflags[si] & SF_HTINY);
    float2 phi = f2(0.f), dE = f2(0.f), dS = f2(0.f);
    float p = 0.f, e1 = 0.f, s1 = 0.f;
    auto flush = [&]() {
        two_add(phi, p); two_add(dE, e1); two_add(dS, s1);
        p = 0.f; e1 = 0.f; s1 = 0.f;
    };
    int cnt = 0;
    const int q0 = min(xl_off[k], capx), q1 = min(xl_off[k + 1], capx);
    if (q0 + lane < q1) {
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
            const bool tiny = A.tiny && (ti || (sflags[sc] & SF_HTINY));
            atom_pair_adj_f(A, dx * dx + dy * dy + dz * dz, xi.w != 0.f, xc.w, li, lc, tiny, p, e1, s1);
            if (++cnt == CHUNK_ADJ) { flush(); cnt = 0; }
        }
    }
    __syncwarp();
    flush();
    phi = sub_two_sum<32>(phi); dE = sub_two_sum<32>(dE); dS = sub_two_sum<32>(dS);
    if (lane != 0) return;
    const int o = site_orig[si];
    dq[o] = R.epstmp * ((double)phi.x + (double)phi.y);
    de[o] = (double)dE.x + (double)dE.y;
    ds[o] = (double)dS.x + (double)dS.y;
}

// erf(alpha r) / r of a squared distance: 2 alpha / sqrt(pi) times the Taylor series of
// erf(x)/x in u = x^2 (Abramowitz & Stegun 7.1.5; 16 terms, exact to rounding for u <= 0.5),
// erf beyond it
__device__ __forceinline__ double erf_over_r(double al, double r2)
{
    const double u = al * al * r2;
    if (u > 0.5) {
        const double r = sqrt(r2);
        return erf(al * r) / r;
    }
    const double c[16] = {1.0, -1.0 / 3, 1.0 / 10, -1.0 / 42, 1.0 / 216, -1.0 / 1320, 1.0 / 9360, -1.0 / 75600,
                          1.0 / 685440, -1.0 / 6894720, 1.0 / 76204800, -1.0 / 918086400, 1.0 / 11975040000.0,
                          -1.0 / 168129561600.0, 1.0 / 2528170444800.0, -1.0 / 40537905408000.0};
    double s = c[15];
#pragma unroll
    for (int k = 14; k >= 0; --k) s = fma(s, u, c[k]);
    return al * NB_TWO_OVER_SQRTPI * s;
}

// Exclusion erf corrections, 1-4 terms and the self energy of n atoms (FP64 coordinates), eight
// lanes per atom; atoms: which (NULL: atom k itself)
#define ADJ_EX_LANES 8
__global__ void __launch_bounds__(128) k_adj_excl14(int n, const int *__restrict__ atoms,
                                                    const int *__restrict__ atom_rep, const RepDev *__restrict__ reps,
                                                    const double *__restrict__ coor, const double *__restrict__ q,
                                                    const double2 *__restrict__ lj, const int *__restrict__ ex_off,
                                                    const int *__restrict__ ex_j, const int *__restrict__ p_off,
                                                    const int *__restrict__ p_j, const double *__restrict__ p_par,
                                                    double *__restrict__ dq, double *__restrict__ de,
                                                    double *__restrict__ ds)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, sub = t & (ADJ_EX_LANES - 1), u = t / ADJ_EX_LANES;
    const bool act = u < n;
    const int a = act ? (atoms ? atoms[u] : u) : 0;
    const RepDev &R = reps[atom_rep[a]];
    const double xa = coor[3 * (size_t)a], ya = coor[3 * (size_t)a + 1], za = coor[3 * (size_t)a + 2];
    double phi = 0, dE = 0, dS = 0;
    for (int k = ex_off[a] + sub; act && k < ex_off[a + 1]; k += ADJ_EX_LANES) {
        const int b = ex_j[k];
        const double rx = xa - coor[3 * (size_t)b], ry = ya - coor[3 * (size_t)b + 1], rz = za - coor[3 * (size_t)b + 2];
        phi -= R.epstmp * q[b] * erf_over_r(R.alphad, rx * rx + ry * ry + rz * rz);
    }
    const int p0 = p_off[a], p1 = p_off[a + 1];
    if (act && p0 + sub < p1) {
        double ea, sa;
        lj_decode(R.arith, lj[a].x, lj[a].y, ea, sa);
        for (int k = p0 + sub; k < p1; k += ADJ_EX_LANES) {
            const int b = p_j[k];
            const double *p = p_par + 3 * (size_t)k;
            const double rx = xa - coor[3 * (size_t)b], ry = ya - coor[3 * (size_t)b + 1], rz = za - coor[3 * (size_t)b + 2];
            const double s2 = 1.0 / (rx * rx + ry * ry + rz * rz), s6 = s2 * s2 * s2;
            if (p[0] > 1e-12) {
                double eb, sb;
                lj_decode(R.arith, lj[b].x, lj[b].y, eb, sb);
                lj_adj(R.arith, p[0] * s6 * s6, p[1] * s6, ea, sa, sb, dE, dS);
            }
            if (fabs(p[2]) > 1e-12 && fabs(q[a]) > 1e-12) phi += p[2] / q[a] * sqrt(s2);
        }
    }
    phi = sub_sum<ADJ_EX_LANES>(phi); dE = sub_sum<ADJ_EX_LANES>(dE); dS = sub_sum<ADJ_EX_LANES>(dS);
    if (!act || sub != 0) return;
    phi -= 2.0 * R.alphad * (NB_TWO_OVER_SQRTPI * 0.5) * R.epstmp * q[a];   // self energy
    dq[a] += phi;
    de[a] += dE;
    ds[a] += dS;
}

// The same for waters whose exclusions are exactly their three pairs (no 1-4 terms): one water
// per thread, each pair's FP64 series once
__global__ void __launch_bounds__(128) k_adj_excl_water(int nW, const int *__restrict__ unit_atom,
                                                        const int *__restrict__ atom_rep,
                                                        const RepDev *__restrict__ reps,
                                                        const double *__restrict__ coor, const double *__restrict__ q,
                                                        double *__restrict__ dq)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nW) return;
    const int a0 = unit_atom[u];
    const RepDev &R = reps[atom_rep[a0]];
    double x[3][3], qs[3], phi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int d = 0; d < 3; ++d) x[k][d] = coor[3 * (size_t)(a0 + k) + d];
        qs[k] = q[a0 + k];
        phi[k] = -2.0 * R.alphad * (NB_TWO_OVER_SQRTPI * 0.5) * qs[k];          // self energy
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const int a = p < 2 ? 0 : 1, b = p < 1 ? 1 : 2;
        const double rx = x[a][0] - x[b][0], ry = x[a][1] - x[b][1], rz = x[a][2] - x[b][2];
        const double w = erf_over_r(R.alphad, rx * rx + ry * ry + rz * rz);
        phi[a] -= qs[b] * w;
        phi[b] -= qs[a] * w;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) dq[a0 + k] += R.epstmp * phi[k];
}

// hi + lo products and sums on the FP32 pipe: a += w * v with w = hi + lo and v exact or hi + lo
__device__ __forceinline__ void two_fma(float2 &a, float2 w, float v)
{
    const float p = w.x * v, e = fmaf(w.x, v, -p);
    two_add(a, p);
    a.y += fmaf(w.y, v, e);
}
__device__ __forceinline__ void two_fma(float2 &a, float2 w, float2 v)
{
    const float p = w.x * v.x, e = fmaf(w.x, v.x, -p);
    two_add(a, p);
    a.y += fmaf(w.x, v.y, fmaf(w.y, v.x, e));
}

// PME: fc * sum(theta * potential grid) at each site, from the real planes k_plane_inv
// leaves in the grid storage (mixed path).  The weights are formed in FP64 and kept as hi + lo
// pairs, as are the sums: 64 conversions and 84 FP64 multiply-adds per site took 70 us for 188,448
// sites on the FP64 pipe, this 38.
__global__ void k_adj_pme_f(int nsite, const int *__restrict__ site_rep, const int *__restrict__ site_orig,
                            const RepDev *__restrict__ reps, const float4 *__restrict__ fr,
                            const float2 *__restrict__ grid, double *__restrict__ dq)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsite) return;
    const RepDev &R = reps[site_rep[s]];
    const float4 f = fr[s];
    const int n1 = R.n1, n2 = R.n2, n3 = R.n3;
    const size_t zs = (size_t)R.n1h * n2 * 2;
    const float *Q = (const float *)(grid + R.g0);
    int i1, i2, i3;
    float w1, w2, w3;
    pme_fr_split(f.x, i1, w1);
    pme_fr_split(f.y, i2, w2);
    pme_fr_split(f.z, i3, w3);
    float2 th[3][4];
    const double w[3] = {(double)w1, (double)w2, (double)w3};
    auto split = [](double v) {
        const float hi = (float)v;
        return f2(hi, (float)(v - (double)hi));
    };
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double u = w[d], u2 = u * u, u3 = u2 * u, m = 1.0 - u;
        th[d][0] = split(m * m * m);                // 6 theta: 1/216 is applied to the sum
        th[d][1] = split(4.0 - 6.0 * u2 + 3.0 * u3);
        th[d][2] = split(1.0 + 3.0 * (u + u2 - u3));
        th[d][3] = split(u3);
    }
    auto wrap = [](int k, int n) { return k < 0 ? k + n : (k >= n ? k - n : k); };
    int xs[4];
#pragma unroll
    for (int t1 = 0; t1 < 4; ++t1) xs[t1] = wrap(i1 - 3 + t1, n1);
    float2 v = f2(0.f);
#pragma unroll
    for (int t3 = 0; t3 < 4; ++t3) {
        const float *P = Q + wrap(i3 - 3 + t3, n3) * zs;
        float2 sy = f2(0.f);
#pragma unroll
        for (int t2 = 0; t2 < 4; ++t2) {
            const float *row = P + wrap(i2 - 3 + t2, n2) * n1;
            float2 sx = f2(0.f);
#pragma unroll
            for (int t1 = 0; t1 < 4; ++t1) two_fma(sx, th[0][t1], row[xs[t1]]);
            two_fma(sy, th[1][t2], sx);
        }
        two_fma(v, th[2][t3], sy);
    }
    dq[site_orig[s]] += R.fcd * ((double)v.x + (double)v.y) * (1.0 / 216.0);
}

// the exclusion and reciprocal parts, formed beside the pair sums, added to them
__global__ void k_adj_add(int64_t n, const double *__restrict__ a, double *__restrict__ o)
{
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k < n) o[k] += a[k];
}

// PME on the plain path: fc * the four plane shares of the potential at each site
__global__ void k_adj_pme_d(int nsite, const int *__restrict__ site_rep, const int *__restrict__ site_orig,
                            const RepDev *__restrict__ reps, const double *__restrict__ phi4, double *__restrict__ dq)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsite) return;
    const double *p = phi4 + 4 * (size_t)s;
    dq[site_orig[s]] += reps[site_rep[s]].fcd * ((p[0] + p[1]) + (p[2] + p[3]));
}

// pair sums of the waters (on sw) and of the other atoms (on sa): the first writes to dq, de, ds
void adjoint_pairs(NbCtx *c, cudaStream_t sw, cudaStream_t sa, double *d_dq, double *d_de, double *d_ds)
{
    const int B = 128, capx = cap_int(c->cap_xl), cap2 = cap_int(c->cap_wl2);
    const bool fp64 = c->precision == MOIL_NB_FP64;
    if (c->nW > 0 && fp64)
        (c->row16 ? k_adj_water<unsigned short> : k_adj_water<int>)<<<(int)((c->nW + 3) / 4), B, 0, sw>>>(
            (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, (const double4 *)c->d_pos, (const double4 *)c->d_woff,
            (const double2 *)c->d_site_lj, c->d_site_flags, c->d_wl1_cnt, c->d_wl1, c->cap_row1, c->d_wl2_off, c->d_wl2, cap2, d_dq, d_de, d_ds);
    else if (c->nW > 0) {
        // lanes per water as the energy kernel (32-bit rows belong to replicas of 65,536 waters or more)
        const int lpw = c->nw_handle <= 4096 ? 32 : 8;
        (!c->row16 ? k_adj_water_f<8, int>
                   : (lpw == 32 ? k_adj_water_f<32, unsigned short> : k_adj_water_f<8, unsigned short>))<<<
            (int)((c->nW * lpw + B - 1) / B), B, 0, sw>>>(
            (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, (const float4 *)c->d_pos, (const float4 *)c->d_woff,
            (const float2 *)c->d_site_lj, c->d_site_flags, c->d_wl1_cnt, c->d_wl1, c->cap_row1, c->d_wl2_off, c->d_wl2,
            cap2, d_dq, d_de, d_ds);
    }
    if (c->nA > 0 && fp64)
        k_adj_atom<<<(int)((c->nA + 3) / 4), B, 0, sa>>>(
            (int)c->nA, (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, (const double4 *)c->d_pos,
            (const double2 *)c->d_site_lj, c->d_site_flags, c->d_xl_off, c->d_xl, capx, d_dq, d_de, d_ds);
    else if (c->nA > 0)
        k_adj_atom_f<<<(int)((c->nA + 3) / 4), B, 0, sa>>>(
            (int)c->nA, (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, (const float4 *)c->d_pos,
            (const float2 *)c->d_site_lj, c->d_site_flags, c->d_xl_off, c->d_xl, capx, d_dq, d_de, d_ds);
}

}  // namespace

void nb_launch_pme_potential(NbCtx *c, double *phi4);

// The mixed path forms the exclusion, 1-4 and reciprocal parts (FP64-pipe and cache-latency bound) on a
// second stream into out2, the non-water atoms' pair sums on a third, beside the waters' pair sums
// (FP32 issue); the plain path, whose kernels all wait for the FP64 pipe, adds them one after the
// other.
int nb_adjoint(NbCtx *c, double *out, double *out2)
{
    cudaStream_t s = c->stream, s2 = out2 ? c->stream2 : s, s3 = out2 ? c->stream3 : s;
    const int B = 128;
    const int64_t na = c->natom;
    if (out2) {
        NB_CUDA_OK(c, cudaEventRecord(c->ev_fork, s));
        NB_CUDA_OK(c, cudaStreamWaitEvent(s2, c->ev_fork, 0));
        NB_CUDA_OK(c, cudaStreamWaitEvent(s3, c->ev_fork, 0));
        NB_CUDA_OK(c, cudaMemsetAsync(out2, 0, sizeof(double) * 3 * na, s2));
    } else {
        adjoint_pairs(c, s, s, out, out + na, out + 2 * na);
    }
    double *x = out2 ? out2 : out;
    const bool fast = c->water_excl_fast && c->nW > 0;
    const int64_t n = fast ? c->nA : na;
    if (n > 0)
        k_adj_excl14<<<(int)((n * ADJ_EX_LANES + 31) / 32), 32, 0, s2>>>(
            (int)n, fast ? c->d_unit_atom + c->nW : nullptr, c->d_atom_rep, c->d_reps, c->d_coor, c->d_q, c->d_lj_d,
            c->d_ex_off, c->d_ex_j, c->d_p14_off, c->d_p14_j, c->d_p14_par, x, x + na, x + 2 * na);
    if (fast)
        k_adj_excl_water<<<(int)((c->nW + 31) / 32), 32, 0, s2>>>((int)c->nW, c->d_unit_atom, c->d_atom_rep, c->d_reps,
                                                                  c->d_coor, c->d_q, x);
    if (c->precision == MOIL_NB_FP64) {
        nb_launch_pme_potential(c, c->d_adj_phi);
        k_adj_pme_d<<<(int)((c->nsite + B - 1) / B), B, 0, s2>>>((int)c->nsite, c->d_site_rep, c->d_site_orig,
                                                               c->d_reps, c->d_adj_phi, x);
    } else {
        k_adj_pme_f<<<(int)((c->nsite + B - 1) / B), B, 0, s2>>>((int)c->nsite, c->d_site_rep, c->d_site_orig,
                                                               c->d_reps, (const float4 *)c->d_fr,
                                                               (const float2 *)c->d_grid, x);
    }
    if (out2) {
        NB_CUDA_OK(c, cudaEventRecord(c->ev_join, s2));
        adjoint_pairs(c, s, s3, out, out + na, out + 2 * na);
        NB_CUDA_OK(c, cudaEventRecord(c->ev_join3, s3));
        NB_CUDA_OK(c, cudaStreamWaitEvent(s, c->ev_join, 0));
        NB_CUDA_OK(c, cudaStreamWaitEvent(s, c->ev_join3, 0));
        k_adj_add<<<(int)((3 * na + 255) / 256), 256, 0, s>>>(3 * na, out2, out);
    }
    NB_CUDA_OK(c, cudaGetLastError());
    return MOIL_NB_OK;
}
