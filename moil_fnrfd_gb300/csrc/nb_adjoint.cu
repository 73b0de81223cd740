// nb_adjoint.cu -- parameter derivatives of the nonbonded energy: dE/dq, dE/deps and
// dE/dsigma per atom (moil_nb_adjoint).  MOIL computes none of them; the oracle's
// ora_adjoint_mi is the reference, itself checked against finite differences.
//
// One evaluation (moil_nb_eval semantics) leaves the lists, the site-ordered positions and
// the PME grid on the device (the real potential planes on the mixed path, the convolved
// spectrum on the plain path, whose inverse plane kernel then gives each site's potential
// shares); these kernels then accumulate, in FP64:
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

template <typename T>
__device__ __forceinline__ double2 lj_of(const void *lj_v, int s)
{
    typedef typename cplx<T>::type T2;
    const T2 v = ((const T2 *)lj_v)[s];
    return make_double2((double)v.x, (double)v.y);
}

// one non-water-semantics site pair (atom_pair of the energy kernels) into site i's sums
template <typename T>
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

// Sum over the W lanes of a subgroup (all lanes of the warp present)
template <int W> __device__ __forceinline__ double lane_sum(double v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, W);
    return v;
}

// one warp per water: W1 (nine site pairs per molecule pair) and W2, the lanes taking the
// entries of both lists in turn
template <typename T, typename E>
__global__ void __launch_bounds__(128) k_adj_water(int nW, const RepDev *__restrict__ reps, const int *__restrict__ site_rep,
                            const int *__restrict__ site_orig, const void *pos_v, const void *woff_v,
                            const void *lj_v, const unsigned *__restrict__ sflags, const int2 *__restrict__ wl1_cnt,
                            const void *__restrict__ wl1, int cap_row, const int *__restrict__ wl2_off,
                            const int *__restrict__ wl2, int cap2, double *__restrict__ dq, double *__restrict__ de,
                            double *__restrict__ ds)
{
    typedef typename vec4<T>::type T4;
    const int lane = threadIdx.x & 31, i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= nW) return;
    const T4 *pos = (const T4 *)pos_v;
    const T4 *woff = (const T4 *)woff_v;
    const RepDev &R = reps[site_rep[3 * i]];
    const T4 oi = pos[3 * i];
    const T4 h1 = woff[3 * i + 1], h2 = woff[3 * i + 2];
    const T hi[3][3] = {{(T)0, (T)0, (T)0}, {h1.x, h1.y, h1.z}, {h2.x, h2.y, h2.z}};
    double phi[3] = {0, 0, 0}, dE[3] = {0, 0, 0}, dS[3] = {0, 0, 0};
    double epsO, sigO;
    const double2 ljO = lj_of<T>(lj_v, 3 * i);
    lj_decode(R.arith, ljO.x, ljO.y, epsO, sigO);
    const int2 c = wl1_cnt[i];
    const int nn = min(c.x, cap_row), n = min(c.x + c.y, cap_row);
    const E *row = (const E *)wl1 + (size_t)i * cap_row;
    const int base = sizeof(E) == 2 ? R.wat0 : 0;   // uint16 entries: offsets from the replica's first water
    for (int v = lane; v < n; v += 32) {
        const int j = base + (int)row[v < nn ? v : cap_row - 1 - (v - nn)];
        const T4 oj = pos[3 * j];
        T dx = oi.x - oj.x, dy = oi.y - oj.y, dz = oi.z - oj.z;
        const T nx = nb_rint(dx * rep_invL<T>(R, 0)), ny = nb_rint(dy * rep_invL<T>(R, 1)),
                nz = nb_rint(dz * rep_invL<T>(R, 2));
        dx = nb_shift(R, 0, dx, nx);
        dy = nb_shift(R, 1, dy, ny);
        dz = nb_shift(R, 2, dz, nz);
        const T r2oo = dx * dx + dy * dy + dz * dz;
        if (r2oo > (T)R.rmax2) continue;
        const T4 j1 = woff[3 * j + 1], j2 = woff[3 * j + 2];
        const T hj[3][3] = {{(T)0, (T)0, (T)0}, {j1.x, j1.y, j1.z}, {j2.x, j2.y, j2.z}};
        const double qj[3] = {(double)oj.w, (double)pos[3 * j + 1].w, (double)pos[3 * j + 2].w};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const double ex = (double)(hi[a][0] + dx - hj[b][0]), ey = (double)(hi[a][1] + dy - hj[b][1]),
                             ez = (double)(hi[a][2] + dz - hj[b][2]);
                const double r = sqrt(ex * ex + ey * ey + ez * ez);
                phi[a] += R.epstmp * qj[b] * erfc(R.alphad * r) / r;
            }
        if (r2oo <= (T)R.rv2) {
            const double s2 = 1.0 / (double)r2oo, s6 = s2 * s2 * s2;
            double ej, sj;
            const double2 ljj = lj_of<T>(lj_v, 3 * j);
            lj_decode(R.arith, ljj.x, ljj.y, ej, sj);
            lj_adj(R.arith, R.w12d * s6 * s6, R.w6d * s6, epsO, sigO, sj, dE[0], dS[0]);
        }
    }
    for (int k = min(wl2_off[i], cap2) + lane; k < min(wl2_off[i + 1], cap2); k += 32) {
        const int s = wl2[k];
        const T4 xj = pos[s];
        const double2 ljj = lj_of<T>(lj_v, s);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const T4 xi = pos[3 * i + a];
            T dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            dx = nb_shift(R, 0, dx, nb_rint(dx * rep_invL<T>(R, 0)));
            dy = nb_shift(R, 1, dy, nb_rint(dy * rep_invL<T>(R, 1)));
            dz = nb_shift(R, 2, dz, nb_rint(dz * rep_invL<T>(R, 2)));
            atom_pair_adj<T>(R, (double)(dx * dx + dy * dy + dz * dz), (double)xi.w, (double)xj.w,
                             lj_of<T>(lj_v, 3 * i + a), ljj, sflags[3 * i + a], sflags[s], phi[a], dE[a], dS[a]);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        phi[a] = lane_sum<32>(phi[a]); dE[a] = lane_sum<32>(dE[a]); dS[a] = lane_sum<32>(dS[a]);
        if (lane != a) continue;
        const int o = site_orig[3 * i + a];
        dq[o] = phi[a];
        de[o] = dE[a];
        ds[o] = dS[a];
    }
}

// one warp per non-water atom over its X list
template <typename T>
__global__ void __launch_bounds__(128) k_adj_atom(int nA, int nW, const RepDev *__restrict__ reps, const int *__restrict__ site_rep,
                           const int *__restrict__ site_orig, const void *pos_v, const void *lj_v,
                           const unsigned *__restrict__ sflags, const int *__restrict__ xl_off,
                           const int *__restrict__ xl, int capx, double *__restrict__ dq, double *__restrict__ de,
                           double *__restrict__ ds)
{
    typedef typename vec4<T>::type T4;
    const int lane = threadIdx.x & 31, k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= nA) return;
    const T4 *pos = (const T4 *)pos_v;
    const int si = 3 * nW + k;
    const RepDev &R = reps[site_rep[si]];
    const T4 xi = pos[si];
    const double2 lji = lj_of<T>(lj_v, si);
    double phi = 0, dE = 0, dS = 0;
    for (int q = min(xl_off[k], capx) + lane; q < min(xl_off[k + 1], capx); q += 32) {
        const int s = xl[q];
        const T4 xj = pos[s];
        T dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        dx = nb_shift(R, 0, dx, nb_rint(dx * rep_invL<T>(R, 0)));
        dy = nb_shift(R, 1, dy, nb_rint(dy * rep_invL<T>(R, 1)));
        dz = nb_shift(R, 2, dz, nb_rint(dz * rep_invL<T>(R, 2)));
        atom_pair_adj<T>(R, (double)(dx * dx + dy * dy + dz * dz), (double)xi.w, (double)xj.w, lji,
                         lj_of<T>(lj_v, s), sflags[si], sflags[s], phi, dE, dS);
    }
    phi = lane_sum<32>(phi); dE = lane_sum<32>(dE); dS = lane_sum<32>(dS);
    if (lane != 0) return;
    const int o = site_orig[si];
    dq[o] = phi;
    de[o] = dE;
    ds[o] = dS;
}

// ---------------------------------------------------------------------------------
// Mixed path: the same sums with FP32 pair arithmetic (the energy kernels' erfc fit and a
// Newton-refined reciprocal square root), summed per site in FP32 over chunks of CHUNK_ADJ list
// entries and flushed into FP64 -- the FP64 pipe of this GPU is a small fraction of the FP32
// one, so per-pair FP64 erfc, square roots and divisions would dominate.  k = kofdie/eps is
// applied to the FP64 potential sums at the end.
#define CHUNK_ADJ 64

// 1/sqrt(r2) to about an ulp: the approximate MUFU value and one Newton step
__device__ __forceinline__ float adj_rsqrt(float r2)
{
    const float y = nb_rsqrt_approx(r2);
    return fmaf(-0.5f * y, fmaf(r2, y * y, -1.f), y);
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

// one non-water-semantics site pair (atom_pair of the energy kernels): q_j erfc(alpha r)/r into
// phi (k applied later), the LJ parts into de, ds of site i (1/(2 eps_i), 1/sigma_i given)
__device__ __forceinline__ void atom_pair_adj_f(const RepDev &R, float r2, float qi, float qj, float2 lji,
                                                float2 ljj, unsigned fi, unsigned fj, float inv2e_i, float sig_i,
                                                float &phi, float &de, float &ds)
{
    const bool hr = !R.arith && R.hvdw0 && ((fi | fj) & SF_HTINY) && r2 < R.re2;
    const bool lj = r2 < R.rv2 && !hr;
    const bool el = r2 < R.rmax2 && qi * qj != 0.f;
    if (!el && !lj) return;
    const float rinv = adj_rsqrt(r2);
    if (el) {
        float ex;
        phi += qj * nb_erfc_ex(R.alpha * r2 * rinv, r2 * R.ex2c, &ex) * rinv;
    }
    if (lj) {
        const float s2 = rinv * rinv, s6 = s2 * s2 * s2;
        float a, b;
        if (!R.arith) {
            a = lji.x * ljj.x * s6 * s6;
            b = lji.y * ljj.y * s6;
        } else {
            const float aa = lji.x * ljj.x, sg = 0.5f * (lji.y + ljj.y);
            float b1 = sg * sg * sg;
            b1 = b1 * b1;
            b = aa * b1 * s6;
            a = aa * b1 * b1 * s6 * s6;
        }
        const float g = 6.f * a - 3.f * b;
        de += (a - b) * inv2e_i;
        if (!R.arith) {
            if (sig_i > 0.f) ds += g / sig_i;
        } else {
            float ej, sj;
            lj_decode_f(1, ljj.x, ljj.y, ej, sj);
            const float sij = 0.5f * (sig_i + sj);
            if (sij > 0.f) ds += g / sij;
        }
    }
}

// LPW lanes per water (FP32 pairs): W1 (nine site pairs per molecule pair, O-O LJ) and W2, the
// lanes taking the entries of both lists in turn; their FP64 sums are added at the end.  One
// water per thread: 249 us for the 460 waters of a small solute system.
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
    const float4 oi = woff[3 * i];
    const float4 h1 = woff[3 * i + 1], h2 = woff[3 * i + 2];
    const float hi[3][3] = {{0.f, 0.f, 0.f}, {h1.x, h1.y, h1.z}, {h2.x, h2.y, h2.z}};
    double phi[3] = {0, 0, 0}, dE[3] = {0, 0, 0}, dS[3] = {0, 0, 0};
    float p[3] = {0.f, 0.f, 0.f}, e3[3] = {0.f, 0.f, 0.f}, s3[3] = {0.f, 0.f, 0.f};
    auto flush = [&]() {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            phi[a] += (double)p[a]; dE[a] += (double)e3[a]; dS[a] += (double)s3[a];
            p[a] = 0.f; e3[a] = 0.f; s3[a] = 0.f;
        }
    };
    float epsO, sigO;
    const float2 ljO = lj[3 * i];
    lj_decode_f(R.arith, ljO.x, ljO.y, epsO, sigO);
    const float inv2eO = epsO > 0.f ? 0.5f / epsO : 0.f, invsO = sigO > 0.f ? 1.f / sigO : 0.f;
    const float alpha = R.alpha, ex2c = R.ex2c, rmax2 = R.rmax2, rv2 = R.rv2, w12 = R.w12, w6 = R.w6;
    const int2 c = wl1_cnt[i];
    const int nn = min(c.x, cap_row), n = act ? min(c.x + c.y, cap_row) : 0;
    const E *row = (const E *)wl1 + (size_t)i * cap_row;
    const int base = sizeof(E) == 2 ? R.wat0 : 0;   // uint16 entries: offsets from the replica's first water
    int cnt = 0;
    for (int v = sub; v < n; v += LPW) {
        const int j = base + (int)row[v < nn ? v : cap_row - 1 - (v - nn)];
        const float4 oj = woff[3 * j];
        float dx = oi.x - oj.x, dy = oi.y - oj.y, dz = oi.z - oj.z;
        dx = nb_shift(R, 0, dx, rintf(dx * R.invL[0]));
        dy = nb_shift(R, 1, dy, rintf(dy * R.invL[1]));
        dz = nb_shift(R, 2, dz, rintf(dz * R.invL[2]));
        const float r2oo = dx * dx + dy * dy + dz * dz;
        if (r2oo > rmax2) continue;
        const float4 j1 = woff[3 * j + 1], j2 = woff[3 * j + 2];
        const float hj[3][3] = {{0.f, 0.f, 0.f}, {j1.x, j1.y, j1.z}, {j2.x, j2.y, j2.z}};
        const float qj[3] = {oj.w, pos[3 * j + 1].w, pos[3 * j + 2].w};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const float ex = hi[a][0] + dx - hj[b][0], ey = hi[a][1] + dy - hj[b][1], ez = hi[a][2] + dz - hj[b][2];
                const float r2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
                const float rinv = adj_rsqrt(r2);
                float exv;
                p[a] += qj[b] * nb_erfc_ex(alpha * r2 * rinv, r2 * ex2c, &exv) * rinv;
            }
        if (r2oo <= rv2) {
            const float ri = adj_rsqrt(r2oo), s2 = ri * ri, s6 = s2 * s2 * s2;
            const float A = w12 * s6 * s6, B = w6 * s6;
            e3[0] += (A - B) * inv2eO;
            s3[0] += (6.f * A - 3.f * B) * invsO;     // sigma_ij = sigma_O for water pairs (both rules)
        }
        if (++cnt == CHUNK_ADJ) { flush(); cnt = 0; }
    }
    flush();
    cnt = 0;
    const int q0 = min(wl2_off[i], cap2), q1 = act ? min(wl2_off[i + 1], cap2) : q0;
    float inv2e[3], sg[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float ea, sa;
        const float2 l = lj[3 * i + a];
        lj_decode_f(R.arith, l.x, l.y, ea, sa);
        inv2e[a] = ea > 0.f ? 0.5f / ea : 0.f;
        sg[a] = sa;
    }
    for (int k = q0 + sub; k < q1; k += LPW) {
        const int s = wl2[k];
        const float4 xj = pos[s];
        const float2 ljj = lj[s];
        const unsigned fj = sflags[s];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float4 xi = pos[3 * i + a];
            float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            dx = nb_shift(R, 0, dx, rintf(dx * R.invL[0]));
            dy = nb_shift(R, 1, dy, rintf(dy * R.invL[1]));
            dz = nb_shift(R, 2, dz, rintf(dz * R.invL[2]));
            atom_pair_adj_f(R, dx * dx + dy * dy + dz * dz, xi.w, xj.w, lj[3 * i + a], ljj, sflags[3 * i + a], fj,
                            inv2e[a], sg[a], p[a], e3[a], s3[a]);
        }
        if (++cnt == CHUNK_ADJ) { flush(); cnt = 0; }
    }
    flush();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        phi[a] = lane_sum<LPW>(phi[a]); dE[a] = lane_sum<LPW>(dE[a]); dS[a] = lane_sum<LPW>(dS[a]);
        if (!act || sub != a) continue;
        const int o = site_orig[3 * i + a];
        dq[o] = R.epstmp * phi[a];
        de[o] = dE[a];
        ds[o] = dS[a];
    }
}

// one warp per non-water atom over its X list (FP32 pairs); one atom per thread: 434 us for 209 atoms
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
    const float4 xi = pos[si];
    const float2 lji = lj[si];
    const unsigned fi = sflags[si];
    float ei, sgi;
    lj_decode_f(R.arith, lji.x, lji.y, ei, sgi);
    const float inv2e = ei > 0.f ? 0.5f / ei : 0.f;
    double phi = 0, dE = 0, dS = 0;
    float p = 0.f, e1 = 0.f, s1 = 0.f;
    int cnt = 0;
    const int q1 = min(xl_off[k + 1], capx);
    for (int q = min(xl_off[k], capx) + lane; q < q1; q += 32) {
        const int s = xl[q];
        const float4 xj = pos[s];
        float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        dx = nb_shift(R, 0, dx, rintf(dx * R.invL[0]));
        dy = nb_shift(R, 1, dy, rintf(dy * R.invL[1]));
        dz = nb_shift(R, 2, dz, rintf(dz * R.invL[2]));
        atom_pair_adj_f(R, dx * dx + dy * dy + dz * dz, xi.w, xj.w, lji, lj[s], fi, sflags[s], inv2e, sgi, p, e1, s1);
        if (++cnt == CHUNK_ADJ) {
            phi += (double)p; dE += (double)e1; dS += (double)s1;
            p = 0.f; e1 = 0.f; s1 = 0.f; cnt = 0;
        }
    }
    phi = lane_sum<32>(phi + (double)p); dE = lane_sum<32>(dE + (double)e1); dS = lane_sum<32>(dS + (double)s1);
    if (lane != 0) return;
    const int o = site_orig[si];
    dq[o] = R.epstmp * phi;
    de[o] = dE;
    ds[o] = dS;
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
    phi = lane_sum<ADJ_EX_LANES>(phi); dE = lane_sum<ADJ_EX_LANES>(dE); dS = lane_sum<ADJ_EX_LANES>(dS);
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

// PME: fc * sum(theta * potential grid) at each site, from the real planes k_plane_inv_f
// leaves in the grid storage (mixed path)
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
    double th[3][4];
    const double w[3] = {(double)w1, (double)w2, (double)w3};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double u = w[d], u2 = u * u, u3 = u2 * u, m = 1.0 - u;
        th[d][0] = m * m * m;                       // 6 theta: 1/216 is applied to the sum
        th[d][1] = 4.0 - 6.0 * u2 + 3.0 * u3;
        th[d][2] = 1.0 + 3.0 * (u + u2 - u3);
        th[d][3] = u3;
    }
    auto wrap = [](int k, int n) { return k < 0 ? k + n : (k >= n ? k - n : k); };
    int xs[4];
#pragma unroll
    for (int t1 = 0; t1 < 4; ++t1) xs[t1] = wrap(i1 - 3 + t1, n1);
    double v = 0.0;
#pragma unroll
    for (int t3 = 0; t3 < 4; ++t3) {
        const float *P = Q + wrap(i3 - 3 + t3, n3) * zs;
        double sy = 0.0;
#pragma unroll
        for (int t2 = 0; t2 < 4; ++t2) {
            const float *row = P + wrap(i2 - 3 + t2, n2) * n1;
            double sx = 0.0;
#pragma unroll
            for (int t1 = 0; t1 < 4; ++t1) sx += th[0][t1] * (double)row[xs[t1]];
            sy += sx * th[1][t2];
        }
        v += sy * th[2][t3];
    }
    dq[site_orig[s]] += R.fcd * v * (1.0 / 216.0);
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

template <typename T>
void adjoint_pairs(NbCtx *c, double *d_dq, double *d_de, double *d_ds)
{
    cudaStream_t s = c->stream;
    const int B = 128;
    if constexpr (sizeof(T) == 4) {
        // lanes per water as the energy kernel (32-bit rows belong to replicas of 65,536 waters or more)
        const int lpw = c->nw_handle <= 4096 ? 32 : 8;
        if (c->nW > 0)
            (!c->row16 ? k_adj_water_f<8, int>
                       : (lpw == 32 ? k_adj_water_f<32, unsigned short> : k_adj_water_f<8, unsigned short>))<<<
                (int)((c->nW * lpw + B - 1) / B), B, 0, s>>>(
                (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, (const float4 *)c->d_pos,
                (const float4 *)c->d_woff, (const float2 *)c->d_site_lj, c->d_site_flags, c->d_wl1_cnt, c->d_wl1,
                c->cap_row1, c->d_wl2_off, c->d_wl2, cap_int(c->cap_wl2), d_dq, d_de, d_ds);
        if (c->nA > 0)
            k_adj_atom_f<<<(int)((c->nA + 3) / 4), B, 0, s>>>(
                (int)c->nA, (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, (const float4 *)c->d_pos,
                (const float2 *)c->d_site_lj, c->d_site_flags, c->d_xl_off, c->d_xl, cap_int(c->cap_xl), d_dq, d_de,
                d_ds);
        return;
    }
    if (c->nW > 0)
        (c->row16 ? k_adj_water<T, unsigned short> : k_adj_water<T, int>)<<<(int)((c->nW + 3) / 4), B, 0, s>>>(
            (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, c->d_pos, c->d_woff, c->d_site_lj,
            c->d_site_flags, c->d_wl1_cnt, c->d_wl1, c->cap_row1, c->d_wl2_off, c->d_wl2, cap_int(c->cap_wl2), d_dq,
            d_de, d_ds);
    if (c->nA > 0)
        k_adj_atom<T><<<(int)((c->nA + 3) / 4), B, 0, s>>>(
            (int)c->nA, (int)c->nW, c->d_reps, c->d_site_rep, c->d_site_orig, c->d_pos, c->d_site_lj,
            c->d_site_flags, c->d_xl_off, c->d_xl, cap_int(c->cap_xl), d_dq, d_de, d_ds);
}

}  // namespace

void nb_launch_pme_potential(NbCtx *c, double *phi4);

int nb_adjoint(NbCtx *c, double *d_dq, double *d_de, double *d_ds)
{
    cudaStream_t s = c->stream;
    const int B = 128;
    if (c->precision == MOIL_NB_FP64) adjoint_pairs<double>(c, d_dq, d_de, d_ds);
    else adjoint_pairs<float>(c, d_dq, d_de, d_ds);
    const bool fast = c->water_excl_fast && c->nW > 0;
    if (fast)
        k_adj_excl_water<<<(int)((c->nW + B - 1) / B), B, 0, s>>>((int)c->nW, c->d_unit_atom, c->d_atom_rep, c->d_reps,
                                                                 c->d_coor, c->d_q, d_dq);
    const int64_t n = fast ? c->nA : c->natom;
    if (n > 0)
        k_adj_excl14<<<(int)((n * ADJ_EX_LANES + B - 1) / B), B, 0, s>>>(
            (int)n, fast ? c->d_unit_atom + c->nW : nullptr, c->d_atom_rep, c->d_reps, c->d_coor, c->d_q, c->d_lj_d,
            c->d_ex_off, c->d_ex_j, c->d_p14_off, c->d_p14_j, c->d_p14_par, d_dq, d_de, d_ds);
    if (c->precision == MOIL_NB_FP64) {
        nb_launch_pme_potential(c, c->d_adj_phi);
        k_adj_pme_d<<<(int)((c->nsite + B - 1) / B), B, 0, s>>>((int)c->nsite, c->d_site_rep, c->d_site_orig,
                                                              c->d_reps, c->d_adj_phi, d_dq);
    } else {
        k_adj_pme_f<<<(int)((c->nsite + B - 1) / B), B, 0, s>>>((int)c->nsite, c->d_site_rep, c->d_site_orig,
                                                              c->d_reps, (const float4 *)c->d_fr,
                                                              (const float2 *)c->d_grid, d_dq);
    }
    NB_CUDA_OK(c, cudaGetLastError());
    return MOIL_NB_OK;
}
